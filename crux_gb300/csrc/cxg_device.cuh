// Device functions shared by the kernels of several translation units:
// the P matrix of one (child edge, component) written into its op record,
// and the FP64 eigensystem of a reversible 4-state Q.
#pragma once

#include <math.h>

#include "cxg_internal.h"

namespace cxg {

// P(t) = max(0, sum_k cube[i][j][k] exp(lambda_k t)) for child c and
// component k of idx = c * kact + k (CxLik.c:258-292), FP64, stored into
// the op record as the plan's precision.  A leaf child (tab >= 0) gets its
// message table instead: row mask = sum over the allowed states j of
// P[i][j], in j order (P times the reference's 0/1 row, CxLik.c:357-374
// with Lik.pyx:1466-1475), in the FP64 table for FP64 plans ([16 masks]
// [kact][4]) and in the record, rounded once to FP32, for FP32 plans.
//
// Four consecutive lanes (q = lane & 3, all four active) share one idx:
// lane q computes exp(lambda_q t) and row i = q, so each lane runs a
// quarter of the serial FP64 work.  Every entry's operations and their
// order are those of one lane doing it all.
__device__ inline void pmat_one(const PmatArgs &a, unsigned idx, unsigned q) {
    const unsigned c = idx / a.kact, k = idx % a.kact;
    const int m = a.model[k];
    // Same association as the reference: ((edgeLen*cmult)*rmult)*wNorm.
    const double wn = a.wnorm_dev ? *a.wnorm_dev : a.wnorm;
    const double t = __dmul_rn(__dmul_rn(__dmul_rn(a.edge_len[c], a.cmult[k]),
                                         a.rmult[k]), wn);
    const double *cube = a.cube + (size_t)m * 64;
    const double *ev = a.eig + (size_t)m * 4;
    const double exq = exp(__dmul_rn(ev[q], t));
    const unsigned gmask = 0xFu << ((threadIdx.x & 31u) & ~3u);
    double ex[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) ex[r] = __shfl_sync(gmask, exq, r, 4);
    const int i = (int)q;
    double P[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        double s = 0.0;
#pragma unroll
        for (int r = 0; r < 4; ++r) s = __dadd_rn(s, __dmul_rn(cube[i * 16 + j * 4 + r], ex[r]));
        P[j] = s < 0.0 ? 0.0 : s;
    }
    const int tb = a.tab[c];
    unsigned char *dst = a.rec + a.dst[c];
    if (tb >= 0) {
        // Message of a leaf with state mask m: the sum over allowed states j
        // of P[i][j], in j order -- exactly P times the reference's 0/1 row.
        // Built incrementally: entry m is entry (m without its highest
        // state h) plus P[i][h], which is the same sum in the same order.
        double T[16];
        T[0] = 0.0;
#pragma unroll
        for (int mk = 1; mk < 16; ++mk) {
            const int h = mk >= 8 ? 3 : mk >= 4 ? 2 : mk >= 2 ? 1 : 0;
            T[mk] = __dadd_rn(T[mk ^ (1 << h)], P[h]);
        }
        if (a.precision == CXG_FP32) {
            // Units of four floats by mask, so that rows of different masks
            // sit in different shared-memory banks: components go in pairs
            // (see Rows in cxg_kernels.cu), the last of an odd number alone.
            const bool lone = (a.kact & 1u) && k + 1 == a.kact;
            float *o = reinterpret_cast<float *>(dst) +
                       (lone ? (size_t)k * 64 + i
                             : (size_t)(k >> 1) * 128 + (i >> 1) * 64 + (i & 1) * 2 + (k & 1u));
#pragma unroll
            for (int mk = 0; mk < 16; ++mk) o[(size_t)mk * 4] = (float)T[mk];
            return;
        }
        double *tt = a.ltab + ((size_t)tb * 16 * a.kact + k) * 4 + i;
#pragma unroll
        for (int mk = 0; mk < 16; ++mk) tt[(size_t)mk * a.kact * 4] = T[mk];
    }
    if (a.precision == CXG_FP32) {
        // By columns, components in pairs (see Rows in cxg_kernels.cu), the
        // last of an odd number alone.
        const bool lone = (a.kact & 1u) && k + 1 == a.kact;
        const unsigned step = lone ? 4 : 8;
        float *o = reinterpret_cast<float *>(dst) +
                   (lone ? (size_t)k * 16 + i : (size_t)(k >> 1) * 32 + i * 2 + (k & 1u));
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j * step] = (float)P[j];
    } else {
        double *o = reinterpret_cast<double *>(dst) + (size_t)k * 16 + i * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = P[j];
    }
}

// The same by sixteen lanes, lane 4 i + j the entry (i, j) and four masks of
// row i's messages: the same products and sums in the same order.
__device__ inline void pmat_one16(const PmatArgs &a, unsigned idx, unsigned l) {
    const unsigned c = idx / a.kact, k = idx % a.kact;
    const int m = a.model[k];
    const double wn = a.wnorm_dev ? *a.wnorm_dev : a.wnorm;
    const double t = __dmul_rn(__dmul_rn(__dmul_rn(a.edge_len[c], a.cmult[k]),
                                         a.rmult[k]), wn);
    const int i = (int)(l >> 2), j = (int)(l & 3u);
    const double *cube = a.cube + (size_t)m * 64 + l * 4;
    const double exq = exp(__dmul_rn(a.eig[(size_t)m * 4 + j], t));
    const unsigned gmask = 0xffffu << (threadIdx.x & 16u);
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
        s = __dadd_rn(s, __dmul_rn(cube[r], __shfl_sync(gmask, exq, r, 4)));
    const double p = s < 0.0 ? 0.0 : s;
    const int tb = a.tab[c];
    unsigned char *dst = a.rec + a.dst[c];
    const bool lone = (a.kact & 1u) && k + 1 == a.kact;
    if (tb >= 0) {
        double P[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) P[q] = __shfl_sync(gmask, p, q, 4);
        // Masks j, j + 4, j + 8, j + 12.
        double T[4];
        T[0] = j & 1 ? P[0] : 0.0;
        if (j & 2) T[0] = __dadd_rn(T[0], P[1]);
        T[1] = __dadd_rn(T[0], P[2]);
        T[2] = __dadd_rn(T[0], P[3]);
        T[3] = __dadd_rn(T[1], P[3]);
        if (a.precision == CXG_FP32) {
            float *o = reinterpret_cast<float *>(dst) +
                       (lone ? (size_t)k * 64 + i
                             : (size_t)(k >> 1) * 128 + (i >> 1) * 64 + (i & 1) * 2 + (k & 1u));
#pragma unroll
            for (int h = 0; h < 4; ++h) o[(size_t)(j + 4 * h) * 4] = (float)T[h];
            return;
        }
        double *tt = a.ltab + ((size_t)tb * 16 * a.kact + k) * 4 + i;
#pragma unroll
        for (int h = 0; h < 4; ++h) tt[(size_t)(j + 4 * h) * a.kact * 4] = T[h];
    }
    if (a.precision == CXG_FP32) {
        float *o = reinterpret_cast<float *>(dst) +
                   (lone ? (size_t)k * 16 + i : (size_t)(k >> 1) * 32 + i * 2 + (k & 1u));
        o[j * (lone ? 4 : 8)] = (float)p;
    } else {
        reinterpret_cast<double *>(dst)[(size_t)k * 16 + l] = p;
    }
}

// ---------------------------------------------------------------------------
// FP64 eigensystem of Q = R Pi (reversible, 4 states): Q is similar to the
// symmetric S = Pi^1/2 Q Pi^-1/2, diagonalised by Jacobi rotations
// (Rutishauser's form), then V = Pi^-1/2 U and V^-1 = U^T Pi^1/2.
// out: [0..3] piNorm, [4] qNorm, [5..68] cube, [69..72] eigenvalues,
// [73] status (0 ok, 1 bad input, 2 no convergence).
// ---------------------------------------------------------------------------

// One warp, all 32 lanes calling; out in memory they can all reach.  Lane
// 4 i + j holds entry (i, j) of S, lane 16 + 4 i + j entry (i, j) of the
// rotations U.  Jacobi by rounds: each round applies two disjoint rotations,
// (0,1)(2,3), then (0,2)(1,3), then (0,3)(1,2).  Disjoint rotations commute
// and neither changes the entries the other's angle is computed from, so
// taking both angles from the round's starting matrix is the same as
// applying them one after the other.
//
// A warp's FP64 instruction takes its SM quarter 64 cycles whether one lane
// or 32 are active, so what counts is the instructions of one lane: an entry
// a lane needs 4 per rotation for S and U (a row a lane: 24), the angle comes
// from two reciprocal square roots (five divisions and roots before), and
// convergence is read from exponents on the integer pipe.
__device__ inline void qdecomp_warp(const double *rtri, const double *pi, double *out) {
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const int i = (int)(lane >> 2) & 3, j = (int)lane & 3;
    const bool in_s = lane < 16;
    double psum = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) psum += pi[k];
    const double pnj = pi[j] / psum;
    if (!__all_sync(kAll, pnj > 0.0)) {
        if (lane == 0) out[73] = 1.0;
        return;
    }
    const double pni = __shfl_sync(kAll, pnj, i);
    const double sqj = sqrt(pnj), sqi = __shfl_sync(kAll, sqj, i);
    // Upper-triangle order of rtri: (0,1) (0,2) (0,3) (1,2) (1,3) (2,3).
    const int lo = min(i, j), hi = max(i, j);
    const double rt = i == j ? 0.0 : rtri[lo == 0 ? hi - 1 : lo + hi];
    // Q = R Pi with zero row sums; qscale = sum over j < i of 2 Q_ij pi_i.
    const double q = rt * pnj, qp = q * pni * 2.0;
    double qscale = 0.0, diag = 0.0;
#pragma unroll
    for (int r = 1; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < r; ++c) qscale += __shfl_sync(kAll, qp, r * 4 + c);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const double x = __shfl_sync(kAll, q, i * 4 + c);
        if (c != i) diag -= x;
    }
    const double slo = i < j ? sqi : sqj, shi = i < j ? sqj : sqi;
    double v = in_s ? (i == j ? diag : rt * slo * shi) : (i == j ? 1.0 : 0.0);
    // The angles take squares of entries: S is brought to [1, 2) by a power of
    // two, so that the units of the rates do not matter, and the eigenvalues
    // back from it at the end.
    const unsigned top = __reduce_max_sync(
        kAll, in_s ? (unsigned)__double2hiint(v) & 0x7ff00000u : 0u) >> 20;
    const int up = max(2046 - (int)top, 1);
    if (in_s) v *= __hiloint2double(up << 20, 0);
    int conv = 0;
    for (int sweep = 0; sweep < 64; ++sweep) {
        // Off-diagonal entries below 2^-61 of the largest on the diagonal (by
        // their exponents; a NaN never converges): what is left out is a
        // change of S by less than a hundredth of an ulp of its entries.
        // (To 2^-67 a call took 37.4 us on average over 400 models, 36.8 now.)
        const unsigned e = (unsigned)__double2hiint(v) & 0x7ff00000u;
        const unsigned off = __reduce_max_sync(kAll, in_s && i != j ? e : 0u);
        const unsigned dg = __reduce_max_sync(kAll, in_s && i == j ? e : 0u);
        if (off == 0u || (off != 0x7ff00000u && off + (62u << 20) <= dg)) {
            conv = 1;
            break;
        }
#pragma unroll
        for (int X = 1; X <= 3; ++X) {  // partner of index a: a ^ X
            const int a = min(j, j ^ X), b = max(j, j ^ X);
            const double app = __shfl_sync(kAll, v, a * 5);
            const double aqq = __shfl_sync(kAll, v, b * 5);
            const double apq2 = 2.0 * __shfl_sync(kAll, v, a * 4 + b);
            // tan 2 phi = 2 apq / (aqq - app), |phi| <= pi / 4:
            // c^2 = (1 + |d| / h) / 2, s = 2 apq sign(d) / (2 c h).
            double c = 1.0, sn = 0.0;
            const double d = aqq - app, h2 = fma(d, d, apq2 * apq2);
            if (h2 > 0.0) {
                const double rh = rsqrt(h2);
                const double c2 = fma(0.5 * fabs(d), rh, 0.5);
                const double rc = rsqrt(c2);
                c = c2 * rc;
                sn = 0.5 * apq2 * rh * rc;
                if (d < 0.0) sn = -sn;
                // To unit length: the rotations stay orthogonal.
                const double dl = -0.5 * fma(c, c, fma(sn, sn, -1.0));
                c = fma(c, dl, c);
                sn = fma(sn, dl, sn);
            }
            // Columns: (lo, hi) -> (c lo - s hi, s lo + c hi).
            double o = __shfl_sync(kAll, v, lane ^ X);
            v = fma(c, v, (j == a ? -sn : sn) * o);
            // Rows of S, with the rotation of row i's pair.
            const double ci = __shfl_sync(kAll, c, i), si = __shfl_sync(kAll, sn, i);
            o = __shfl_sync(kAll, v, lane ^ (X << 2));
            const double w = fma(ci, v, ((i ^ X) < i ? si : -si) * o);
            if (in_s) v = (i ^ j) == X ? 0.0 : w;
        }
    }
    if (lane < 4) out[lane] = pnj;
    if (lane == 0) out[4] = 1.0 / qscale;
    // cube[i][j][k] = V[i][k] V^-1[k][j] with V = Pi^-1/2 U, V^-1 = U^T Pi^1/2:
    // two k a lane.
    const double isq = 1.0 / sqi;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int k = (in_s ? 0 : 2) + t;
        const double uik = __shfl_sync(kAll, v, 16 + i * 4 + k);
        const double ujk = __shfl_sync(kAll, v, 16 + j * 4 + k);
        out[5 + i * 16 + j * 4 + k] = (uik * isq) * (ujk * sqj);
    }
    if (in_s && i == j) out[69 + i] = scalbn(v, 1023 - up);
    if (lane == 0) out[73] = conv ? 0.0 : 2.0;
}

}  // namespace cxg
