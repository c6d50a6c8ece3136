// element_mma.cuh -- the contractions of one element on FP64 tensor-core fragments (dmma.cuh).
//
// All of them are products of element data with a shape table, summed over quadrature points or
// nodes.  The element data is the left factor (its 8 x 4 fragments are formed by the lanes, on the
// fly, once for every right factor), columns of the local system are rows of the fragment, and
// the values are consumed where they come out.  A job is a block of 8 columns and belongs to one
// warp; there is no exchange between warps and no barrier inside.
// Bound by shared-memory reads of the left factors and by the tensor pipe in like measure; before, as
// register tiles of scalar multiply-adds (5 x 2 outputs a thread), the reads alone took five
// times the multiply-adds' time.
#pragma once
#include "dmma.cuh"

namespace hdgx {

// smallest value >= x that is 4 modulo 8: as the stride (in doubles) between the four columns or rows
// that the lanes of a fragment read together, it keeps them on different banks
__host__ __device__ constexpr int pad4(int x) { return x + ((4 - x % 8) + 8) % 8; }

// For every column c < NCOL of a local matrix and every component a, over rows r < NPV:
//   out(a, r, c) = sum_{k < KV} left_v(c, k, a) right_v(r, k) + sum_{k < KF} left_f(c, k, a) right_f(r, k)
// left_*(c, k, w) fills w[0 .. NCU) for all a; store(c, a, r, value) consumes.
//
// Here and below, lanes past the last column, row or point read the last one instead (what comes of it
// is not stored, or its factor is set to zero): a branch around a read keeps the reads from being
// issued together, which cost more than the products.
template <int NCU, int NPV, int KV, int KF, int NCOL, int NT, class LV, class RV, class LF, class RF, class ST>
__device__ __forceinline__ void column_product(LV left_v, RV right_v, LF left_f, RF right_f, ST store) {
    constexpr int TN = (NPV + 7) / 8, NW = NT / 32;
    const int lane = threadIdx.x & 31, m = lane >> 2, q = lane & 3;
    for (int ct = threadIdx.x >> 5; ct < (NCOL + 7) / 8; ct += NW) {
        const bool in = NCOL % 8 == 0 || 8 * ct + m < NCOL;
        const int c = in ? 8 * ct + m : NCOL - 1;
        double acc[NCU][TN][2];
#pragma unroll
        for (int a = 0; a < NCU; a++)
#pragma unroll
            for (int t = 0; t < TN; t++) acc[a][t][0] = acc[a][t][1] = 0.0;
        auto accumulate = [&](const double (&w)[NCU], const double (&p)[TN]) {
#pragma unroll
            for (int a = 0; a < NCU; a++)
#pragma unroll
                for (int t = 0; t < TN; t++) dmma(acc[a][t], w[a], p[t]);
        };
#pragma unroll 2
        for (int s = 0; s < (KV + 3) / 4; s++) {
            const bool ink = KV % 4 == 0 || 4 * s + q < KV;
            const int k = ink ? 4 * s + q : KV - 1;
            double w[NCU] = {}, p[TN];
            left_v(c, k, w);
#pragma unroll
            for (int t = 0; t < TN; t++) p[t] = right_v(NPV % 8 == 0 || 8 * t + m < NPV ? 8 * t + m : NPV - 1, k);
            if constexpr (KV % 4 != 0) {
#pragma unroll
                for (int a = 0; a < NCU; a++) w[a] = ink ? w[a] : 0.0;
#pragma unroll
                for (int t = 0; t < TN; t++) p[t] = ink ? p[t] : 0.0;
            }
            accumulate(w, p);
        }
#pragma unroll 2
        for (int s = 0; s < (KF + 3) / 4; s++) {
            const bool ink = KF % 4 == 0 || 4 * s + q < KF;
            const int k = ink ? 4 * s + q : KF - 1;
            double w[NCU] = {}, p[TN];
            left_f(c, k, w);
#pragma unroll
            for (int t = 0; t < TN; t++) p[t] = right_f(NPV % 8 == 0 || 8 * t + m < NPV ? 8 * t + m : NPV - 1, k);
            if constexpr (KF % 4 != 0) {
#pragma unroll
                for (int a = 0; a < NCU; a++) w[a] = ink ? w[a] : 0.0;
#pragma unroll
                for (int t = 0; t < TN; t++) p[t] = ink ? p[t] : 0.0;
            }
            accumulate(w, p);
        }
        if (in) {
#pragma unroll
            for (int a = 0; a < NCU; a++)
#pragma unroll
                for (int t = 0; t < TN; t++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int r = 8 * t + 2 * q + h;
                        if (NPV % 8 == 0 || r < NPV) store(c, a, r, acc[a][t][h]);
                    }
        }
    }
}

// The face integrals by face: for every column c < NCOL, face j, face node n and component a
//   out(a, n, j, c) = sum_g left(c, j, g, a) fg(n, g)
template <int NCU, int NPF, int NFE, int NGF, int NCOL, int NT, class LF, class ST>
__device__ __forceinline__ void face_product(const double *__restrict__ fg, LF left, ST store) {
    constexpr int TN = (NPF + 7) / 8, NW = NT / 32;
    const int lane = threadIdx.x & 31, m = lane >> 2, q = lane & 3;
    constexpr int NJ = (NCOL + 7) / 8 * NFE;                 // a job is a face of a block of 8 columns
    for (int job = threadIdx.x >> 5; job < NJ; job += NW) {
        const int j = job % NFE, c0 = 8 * (job / NFE) + m;
        const bool in = NCOL % 8 == 0 || c0 < NCOL;
        const int c = in ? c0 : NCOL - 1;
        double acc[NCU][TN][2];
#pragma unroll
        for (int a = 0; a < NCU; a++)
#pragma unroll
            for (int t = 0; t < TN; t++) acc[a][t][0] = acc[a][t][1] = 0.0;
#pragma unroll
        for (int s = 0; s < (NGF + 3) / 4; s++) {
            const bool ing = NGF % 4 == 0 || 4 * s + q < NGF;
            const int g = ing ? 4 * s + q : NGF - 1;
            double w[NCU] = {};
            left(c, j, g, w);
            if constexpr (NGF % 4 != 0) {
#pragma unroll
                for (int a = 0; a < NCU; a++) w[a] = ing ? w[a] : 0.0;
            }
#pragma unroll
            for (int t = 0; t < TN; t++) {
                double p = fg[(NPF % 8 == 0 || 8 * t + m < NPF ? 8 * t + m : NPF - 1) + NPF * g];
                if constexpr (NGF % 4 != 0) p = ing ? p : 0.0;
#pragma unroll
                for (int a = 0; a < NCU; a++) dmma(acc[a][t], w[a], p);
            }
        }
        if (in) {
#pragma unroll
            for (int a = 0; a < NCU; a++)
#pragma unroll
                for (int t = 0; t < TN; t++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int n = 8 * t + 2 * q + h;
                        if (NPF % 8 == 0 || n < NPF) store(c, a, n, j, acc[a][t][h]);
                    }
        }
    }
}

// Stores of the outputs, which the element does not read again, past L1: it is left to the tables and to
// spilled registers (3D p = 2, two CTAs in 225 KB of shared memory: 1,060 -> 900 us on 3,072 elements).
__device__ __forceinline__ void store_out(double *p, double v) {
    asm volatile("st.global.L1::no_allocate.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
// two values to consecutive addresses, as one 16-byte store where `wide` says that they are aligned to it
__device__ __forceinline__ void store2(double *p, double v0, double v1, bool wide) {
    if (wide) {
        asm volatile("st.global.L1::no_allocate.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v0), "d"(v1) : "memory");
    } else {
        store_out(p, v0);
        store_out(p + 1, v1);
    }
}

// The trace Jacobian, face by face: for columns c < NH and the unknowns o = (a, n) of face j
//   AE(o, j, c) = sum_{k < K} left(c, k, j) right(k, o, j) + sum_{a', g} face(c, j, g, a') [a == a'] fg(n, g)
// (the second sum is H - GK_q Mi E, whose left factor depends on the component).  A job is 8 columns and
// a face; on(c, j) says whether the second sum has anything for column c.
template <int NCU, int NPF, int NFE, int NGF, int NH, int K, int NT, class FL, class FR, class FF, class FO>
__device__ __forceinline__ void trace_jacobian(const double *__restrict__ fg, double *ae, bool wide, FL left, FR right, FF face,
                                               FO on) {
    constexpr int KQ = NPF * NCU, OT = (KQ + 7) / 8, NJ = (NH + 7) / 8 * NFE, NW = NT / 32;
    const int lane = threadIdx.x & 31, m = lane >> 2, q = lane & 3;
    for (int job = threadIdx.x >> 5; job < NJ; job += NW) {
        const int j = job % NFE, c0 = 8 * (job / NFE) + m;
        const bool in = NH % 8 == 0 || c0 < NH;
        const int c = in ? c0 : NH - 1;
        double acc[OT][2];
#pragma unroll
        for (int t = 0; t < OT; t++) acc[t][0] = acc[t][1] = 0.0;
#pragma unroll 4
        for (int s = 0; s < (K + 3) / 4; s++) {
            const bool ink = K % 4 == 0 || 4 * s + q < K;
            const int k = ink ? 4 * s + q : K - 1;
            double l = left(c, k, j), r[OT];
#pragma unroll
            for (int t = 0; t < OT; t++) r[t] = right(k, KQ % 8 == 0 || 8 * t + m < KQ ? 8 * t + m : KQ - 1, j);
            if constexpr (K % 4 != 0) {
                l = ink ? l : 0.0;
#pragma unroll
                for (int t = 0; t < OT; t++) r[t] = ink ? r[t] : 0.0;
            }
#pragma unroll
            for (int t = 0; t < OT; t++) dmma(acc[t], l, r[t]);
        }
        if (__any_sync(0xffffffffu, in && on(c, j))) {
#pragma unroll
            for (int s = 0; s < (NGF + 3) / 4; s++) {
                const bool ing = NGF % 4 == 0 || 4 * s + q < NGF;
                const int g = ing ? 4 * s + q : NGF - 1;
                double w[NCU] = {};
                face(c, j, g, w);
                if constexpr (NGF % 4 != 0) {
#pragma unroll
                    for (int a = 0; a < NCU; a++) w[a] = ing ? w[a] : 0.0;
                }
#pragma unroll
                for (int t = 0; t < OT; t++) {
                    const int o = KQ % 8 == 0 || 8 * t + m < KQ ? 8 * t + m : KQ - 1, n = o / NCU, ao = o - NCU * n;
                    double p = fg[n + NPF * g];
                    if constexpr (NGF % 4 != 0) p = ing ? p : 0.0;
#pragma unroll
                    for (int a = 0; a < NCU; a++) dmma(acc[t], w[a], a == ao ? p : 0.0);
                }
            }
        }
        if (in) {
            double *to = ae + NH * c + KQ * j + 2 * q;
#pragma unroll
            for (int t = 0; t < OT; t++) {
                if (KQ % 2 == 0) {
                    if (KQ % 8 == 0 || 8 * t + 2 * q < KQ) store2(to + 8 * t, acc[t][0], acc[t][1], wide);
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        if (8 * t + 2 * q + h < KQ) store_out(to + 8 * t + h, acc[t][h]);
                }
            }
        }
    }
}

// The q rows of DUDG_DUH: for column k = (b, f), component a, direction d, node r
//   dd(r, a, d, k) = sum_s MiC(r, s, d) dlu(s, a, k) - (a == b) MiE(r, f, d)
// R: dlu [LDR, NH], dd: row (r, a, d) of column k at dd[NQ k + r + NPV (a + NCU d)].  Rows of the
// fragments are (a, k); the right factor Mi C stays in registers for every job, and so do a lane's
// offsets in the output: with them computed per value, the index arithmetic took most of the time.
template <int NPV, int ND, int NCU, int NDF, int NH, int LDR, int NQ, int NT>
__device__ __forceinline__ void q_rows(const double *R, const double *MiC, const double *MiE, double *dd, bool wide) {
    constexpr int KS = (NPV + 3) / 4, OT = (NPV * ND + 7) / 8, TO = OT <= 4 ? OT : 4, CT = (NCU * NH + 7) / 8, NW = NT / 32;
    const int lane = threadIdx.x & 31, m = lane >> 2, q = lane & 3;
    for (int o0 = 0; o0 < 8 * OT; o0 += 8 * TO) {
        double right[TO][KS];
        int to[TO][2], me[TO][2];                                // offsets in a column of dd, in MiE; -1: no output
#pragma unroll
        for (int t = 0; t < TO; t++) {
            const int o = o0 + 8 * t + m, r = o % NPV, d = o / NPV;
#pragma unroll
            for (int s = 0; s < KS; s++)
                right[t][s] = o < NPV * ND && 4 * s + q < NPV ? MiC[r + NPV * (4 * s + q + NPV * d)] : 0.0;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int oo = o0 + 8 * t + 2 * q + h, rr = oo % NPV, de = oo / NPV;
                to[t][h] = oo < NPV * ND ? rr + NPV * NCU * de : -1;
                me[t][h] = oo < NPV * ND ? rr + NPV * NDF * de : 0;
            }
        }
        for (int job = threadIdx.x >> 5; job < CT; job += NW) {
            const int ak = 8 * job + m;
            const bool in = (NCU * NH) % 8 == 0 || ak < NCU * NH;
            const int k = in ? ak / NCU : 0, a = in ? ak - NCU * k : 0, f = k / NCU;
            const bool same = in && a == k - NCU * f;
            double acc[TO][2], left[KS];
#pragma unroll
            for (int s = 0; s < KS; s++)
                left[s] = R[LDR * k + NPV * a + (NPV % 4 == 0 || 4 * s + q < NPV ? 4 * s + q : NPV - 1)];
            if constexpr (NPV % 4 != 0) left[KS - 1] = 4 * (KS - 1) + q < NPV ? left[KS - 1] : 0.0;
#pragma unroll
            for (int t = 0; t < TO; t++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const double v = MiE[me[t][h] + NPV * f];    // read without a branch: one took half the time
                    acc[t][h] = same ? -v : 0.0;
                }
#pragma unroll
            for (int s = 0; s < KS; s++)
#pragma unroll
                for (int t = 0; t < TO; t++) dmma(acc[t], left[s], right[t][s]);
            if (in) {
                double *col = dd + (size_t)NQ * k + NPV * a;
#pragma unroll
                for (int t = 0; t < TO; t++) {
                    if (NPV % 2 == 0) {
                        if (to[t][0] >= 0) store2(col + to[t][0], acc[t][0], acc[t][1], wide);
                    } else {
                        if (to[t][0] >= 0) store_out(col + to[t][0], acc[t][0]);
                        if (to[t][1] >= 0) store_out(col + to[t][1], acc[t][1]);
                    }
                }
            }
        }
    }
}

}  // namespace hdgx
