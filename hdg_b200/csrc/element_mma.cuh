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
template <int NCU, int NPV, int KV, int KF, int NCOL, int NT, class LV, class RV, class LF, class RF, class ST>
__device__ __forceinline__ void column_product(LV left_v, RV right_v, LF left_f, RF right_f, ST store) {
    constexpr int TN = (NPV + 7) / 8, NW = NT / 32;
    const int lane = threadIdx.x & 31, m = lane >> 2, q = lane & 3;
    for (int ct = threadIdx.x >> 5; ct < (NCOL + 7) / 8; ct += NW) {
        const int c = 8 * ct + m;
        const bool in = c < NCOL;
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
            const int k = 4 * s + q;
            double w[NCU] = {}, p[TN];
            const bool ink = KV % 4 == 0 || k < KV;
            if (in && ink) left_v(c, k, w);
#pragma unroll
            for (int t = 0; t < TN; t++) p[t] = ink && (NPV % 8 == 0 || 8 * t + m < NPV) ? right_v(8 * t + m, k) : 0.0;
            accumulate(w, p);
        }
#pragma unroll 2
        for (int s = 0; s < (KF + 3) / 4; s++) {
            const int k = 4 * s + q;
            double w[NCU] = {}, p[TN];
            const bool ink = KF % 4 == 0 || k < KF;
            if (in && ink) left_f(c, k, w);
#pragma unroll
            for (int t = 0; t < TN; t++) p[t] = ink && (NPV % 8 == 0 || 8 * t + m < NPV) ? right_f(8 * t + m, k) : 0.0;
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
        const int j = job % NFE, c = 8 * (job / NFE) + m;
        const bool in = c < NCOL;
        double acc[NCU][TN][2];
#pragma unroll
        for (int a = 0; a < NCU; a++)
#pragma unroll
            for (int t = 0; t < TN; t++) acc[a][t][0] = acc[a][t][1] = 0.0;
#pragma unroll
        for (int s = 0; s < (NGF + 3) / 4; s++) {
            const int g = 4 * s + q;
            double w[NCU] = {};
            const bool ing = NGF % 4 == 0 || g < NGF;
            if (in && ing) left(c, j, g, w);
#pragma unroll
            for (int t = 0; t < TN; t++) {
                const double p = ing && (NPF % 8 == 0 || 8 * t + m < NPF) ? fg[8 * t + m + NPF * g] : 0.0;
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

// Output tiles per job of matrix_product: the count (at most 6) that leaves the busiest warp the least
// to do, a tile counted as one and the left fragment as one more.
__host__ __device__ constexpr int tiles_per_job(int ct, int ot, int nw) {
    int best = 1, cost = 1 << 30;
    for (int t = 1; t <= 6 && t <= ot; t++) {
        const int c = (ct * ((ot + t - 1) / t) + nw - 1) / nw * (t + 1);
        if (c <= cost) { best = t; cost = c; }
    }
    return best;
}

// out(c, o) = init(c, o) + sum_{k < K} left(c, k) right(k, o) for c < NCOL, o < NOUT, in jobs of 8
// columns by a few tiles of 8 outputs.  store(c, o, v0, v1, n) consumes the outputs o and (n == 2) o + 1;
// init is read when the job begins.  first: the warp that takes job 0 (several products share the
// warps evenly); returns the next one's.
template <int NCOL, int NOUT, int K, int NT, class FI, class FL, class FR, class ST>
__device__ __forceinline__ int matrix_product(int first, FI init, FL left, FR right, ST store) {
    constexpr int CT = (NCOL + 7) / 8, OT = (NOUT + 7) / 8, NW = NT / 32, TO = tiles_per_job(CT, OT, NW),
                  GO = (OT + TO - 1) / TO;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m = lane >> 2, q = lane & 3;
    for (int job = (w + NW - first) % NW; job < CT * GO; job += NW) {
        const int c = 8 * (job % CT) + m, o0 = 8 * TO * (job / CT);
        const bool in = NCOL % 8 == 0 || c < NCOL;
        double acc[TO][2], ini[TO][2];
#pragma unroll
        for (int t = 0; t < TO; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int o = o0 + 8 * t + 2 * q + h;
                ini[t][h] = in && (NOUT % (8 * TO) == 0 || o < NOUT) ? init(c, o) : 0.0;
                acc[t][h] = 0.0;
            }
#pragma unroll 4
        for (int s = 0; s < (K + 3) / 4; s++) {
            const int k = 4 * s + q;
            const bool ink = K % 4 == 0 || k < K;
            const double l = in && ink ? left(c, k) : 0.0;
#pragma unroll
            for (int t = 0; t < TO; t++) {
                const int o = o0 + 8 * t + m;
                const double r = ink && (NOUT % (8 * TO) == 0 || o < NOUT) ? right(k, o) : 0.0;
                dmma(acc[t], l, r);
            }
        }
        if (in) {
#pragma unroll
            for (int t = 0; t < TO; t++) {
                const int o = o0 + 8 * t + 2 * q;
                if (NOUT % (8 * TO) == 0 || o < NOUT)
                    store(c, o, acc[t][0] + ini[t][0], acc[t][1] + ini[t][1], NOUT % 2 == 0 || o + 1 < NOUT ? 2 : 1);
            }
        }
    }
    return (first + CT * GO) % NW;
}

// two values to consecutive addresses, as one 16-byte store where `wide` says that they are aligned to it
__device__ __forceinline__ void store2(double *p, double v0, double v1, bool wide) {
    if (wide) {
        *reinterpret_cast<double2 *>(p) = make_double2(v0, v1);
    } else {
        p[0] = v0;
        p[1] = v1;
    }
}

}  // namespace hdgx
