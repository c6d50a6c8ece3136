// schur_mma.cuh -- the local (u,q) Schur complement of given blocks (kernel/schur_uq.c:42-191,
// kernel/schur_primal.m:52-150) for the element shapes of the elemental kernel, on FP64 tensor-core
// fragments.  One CTA per element.
//
// Both coupling operators, B = dRu/dq and GK_q = dRh/dq, meet only Mi C, Mi E and Mi Rq: their blocks are
// read from global memory once, as right factors, and meet all three in one pass (coupled_product),
//   SD = D + B Mi C,  R = [Ru - B Mi Rq | B Mi E - F],
//   G' = GK_u + GK_q Mi C,  AE <- H - GK_q Mi E,
// and after the solve AE += G' dlu, FE = Rh - GK_q Mi Rq - G' du (DUDG_DUH is never read back).
// The blocks are a caller's: M and SD are eliminated without pivoting together with one fixed right-hand side
// (probe_rhs), and again with partial pivoting when that is not solved to rounding.
// Bound by the reads of the blocks and the elimination; 2D p = 3, 4,050 elements (190 KB each):
// 3.41 -> 0.347 ms, of which the DRAM traffic takes 0.12 ms at 6.5 TB/s.
#pragma once
#include "element_mma.cuh"
#include "hdgx_common.cuh"

namespace hdgx {

struct SchurParams {
    int nd, npv, ncu, nc, ndf, ne, qform;   // qform 1: (u,q) form, 0: u only
    const double *M, *C, *E, *BD, *F, *GK, *H, *Rq, *Ru, *Rh;
    double *DUDG, *DUDG_DUH, *AE, *FE;
    int *status;
    int tile;
};

// For block row r < ROWS and component b, with X(j, d, col) = [Mi C | Mi E | Mi Rq of component b]:
//   out(b, col, r) = init + sum_{j, d} gq(r, j, b, d) X(j, d, col)
// where init(b, col, r, sign) gives the place of a value in global memory and its sign (0: nothing).
// gq: [ROWS, NPV, NCU, ND] in global memory.  Mi: Mi C [NPV, NPV, ND], Mi E [NPV, NDF, ND], Mi Rq [NPV, NCU, ND]
// one after another.  A job is a component and 8 rows; first as in the caller's job list.
template <int ND, int NPV, int NCU, int NDF, int ROWS, int NT, class FI, class ST>
__device__ __forceinline__ int coupled_product(int first, const double *__restrict__ gq, const double *Mi, FI init, ST store) {
    constexpr int K = NPV * ND, KS = (K + 3) / 4, COLS = NPV + NDF + 1, CT = (COLS + 7) / 8, RT = (ROWS + 7) / 8,
                  NW = NT / 32, NJ = NCU * RT;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m = lane >> 2, q = lane & 3;
    int base[CT], step[CT];                                      // a lane's column in Mi, and from one d to the next
    bool res[CT];
#pragma unroll
    for (int t = 0; t < CT; t++) {
        const int col = 8 * t + m < COLS ? 8 * t + m : COLS - 1;
        res[t] = col == COLS - 1;
        base[t] = col < NPV ? NPV * col
                            : (col < NPV + NDF ? NPV * NPV * ND + NPV * (col - NPV) : NPV * (NPV + NDF) * ND);
        step[t] = col < NPV ? NPV * NPV : (col < NPV + NDF ? NPV * NDF : NPV * NCU);
    }
    for (int job = (w + NW - first) % NW; job < NJ; job += NW) {
        const int b = job % NCU, r0 = 8 * (job / NCU);
        const int rl = ROWS % 8 == 0 || r0 + m < ROWS ? r0 + m : ROWS - 1;
        double g[KS], acc[CT][2], ini[CT][2];
#pragma unroll
        for (int s = 0; s < KS; s++) {
            const int k = 4 * s + q < K ? 4 * s + q : K - 1, d = k / NPV, j = k - NPV * d;
            g[s] = __ldg(gq + rl + (size_t)ROWS * (j + NPV * (b + NCU * d)));
        }
#pragma unroll
        for (int t = 0; t < CT; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = ROWS % 8 == 0 || r0 + 2 * q + h < ROWS ? r0 + 2 * q + h : ROWS - 1;
                double sign;
                const double v = __ldg(init(b, 8 * t + m < COLS ? 8 * t + m : COLS - 1, r, sign));
                ini[t][h] = sign == 0.0 ? 0.0 : sign * v;
                acc[t][h] = 0.0;
            }
#pragma unroll
        for (int s = 0; s < KS; s++) {
            const bool ink = K % 4 == 0 || 4 * s + q < K;
            const int k = ink ? 4 * s + q : K - 1, d = k / NPV, j = k - NPV * d;
            const double gs = ink ? g[s] : 0.0;
#pragma unroll
            for (int t = 0; t < CT; t++) {
                double x = Mi[base[t] + (res[t] ? NPV * b : 0) + j + step[t] * d];
                if constexpr (K % 4 != 0) x = ink ? x : 0.0;
                dmma(acc[t], x, gs);
            }
        }
#pragma unroll
        for (int t = 0; t < CT; t++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int col = 8 * t + m, r = r0 + 2 * q + h;
                if (col < COLS && (ROWS % 8 == 0 || r < ROWS)) store(b, col, r, acc[t][h] + ini[t][h]);
            }
    }
    return (first + NJ) % NW;
}

template <int ND, int NPV, int NCU, int NDF>
struct SchurShape {
    static constexpr int ev2(int x) { return (x + 1) / 2 * 2; }
    static constexpr int NC = NCU * (ND + 1), NU = NPV * NCU, NH = NCU * NDF, NQ = NPV * NC;
    static constexpr int LDR = pad4(NU), SG = pad4(NH), NX = NPV * ND + NDF * ND + NCU * ND;   // and one probe_rhs
    static constexpr int o_M = 0, o_Mi = o_M + NPV * NPV, o_SD = o_Mi + NPV * (NX + 1), o_R = ev2(o_SD + NU * NU),
                         o_G = o_R + LDR * (2 + NH), o_pub = ev2(o_G + NU * SG),
                         o_part = o_pub + BlockGJ<NU, 1, 32>::pub_doubles, o_red = o_part + NCU * NH,
                         o_int = o_red + 32, doubles = o_int;
    static constexpr int i_ord = 0, i_face = NU, i_var = i_face + NPV, i_slot = i_var + NU, i_bad = i_slot + 4, ints = i_bad + 2;
    static constexpr size_t bytes = sizeof(double) * doubles + sizeof(int) * ints;
    // As many CTAs as shared memory holds, up to six, and threads so that their registers suffice (fewer threads leave the
    // elimination to fewer warps).  In us with two thirds of the threads / these / a third more where there is room / fewer
    // CTAs of as many threads: 2D p = 1, 16,200 elements, 328 / 293 / 268 / 353; p = 2, 9,800, 380 / 336 / 328 / 366;
    // p = 3, 4,050, 366 / 346 / 334 / 377; p = 4, 1,800, 564 / 414 / 419 / 551; 3D p = 1, 4,374, 358 / 326 / 314 / 260; p = 2, 1,296,
    // 1,028 / 576 / 574 / 577.
    static constexpr int blocks = bytes <= 36 * 1024 ? 6 : (bytes <= 56 * 1024 ? 4 : (bytes <= 74 * 1024 ? 3 : (bytes <= 113 * 1024 ? 2 : 1)));
    static constexpr int threads = blocks == 6 ? 96 : (blocks == 4 ? 128 : (blocks == 3 ? 192 : 256));
};

template <int ND, int NPV, int NCU, int NDF>
__global__ void __launch_bounds__(SchurShape<ND, NPV, NCU, NDF>::threads, SchurShape<ND, NPV, NCU, NDF>::blocks)
    schur_uq_mma_kernel(const __grid_constant__ SchurParams P) {
    using S = SchurShape<ND, NPV, NCU, NDF>;
    constexpr int NT = S::threads, NU = S::NU, NH = S::NH, NQ = S::NQ, LDR = S::LDR, SG = S::SG, NX = S::NX;
    static_assert(NQ >= NH, "DUDG_DUH has room for a trace Jacobian");
    extern __shared__ __align__(16) double sm[];
    double *sM = sm + S::o_M, *sMi = sm + S::o_Mi, *sMiE = sMi + NPV * NPV * ND, *sMiRq = sMiE + NPV * NDF * ND;
    double *sSD = sm + S::o_SD, *sR = sm + S::o_R, *sG = sm + S::o_G, *pub = sm + S::o_pub, *part = sm + S::o_part;
    // the published blocks' place also holds B Mi Rq by component before SD's elimination, and what a pivoted one works with
    double *partu = pub, *fall = pub;
    double *red = sm + S::o_red;
    int *si = reinterpret_cast<int *>(sm + S::o_int), *ord = si + S::i_ord, *face = si + S::i_face, *var = si + S::i_var,
        *slot = si + S::i_slot, *sbad = si + S::i_bad;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, m = lane >> 2, q = lane & 3;
    for (int e = blockIdx.x; e < P.ne; e += gridDim.x) {
        const double *BD = P.BD + (size_t)e * NU * NQ, *F = P.F + (size_t)e * NU * NH, *GK = P.GK + (size_t)e * NH * NQ;
        const double *H = P.H + (size_t)e * NH * NH, *C = P.C + (size_t)e * NPV * NPV * ND;
        double *dd = P.DUDG_DUH + (size_t)e * NQ * NH, *ae = P.AE + (size_t)e * NH * NH;
        const bool wide = (((size_t)P.DUDG_DUH | (size_t)P.AE) & 15) == 0;
        double *ah = ae;                                 // where H - GK_q Mi E goes
        bool pivot_m = false, pivot_sd = false;          // an elimination failed its check: again, with pivoting
    element:
        if (tid == 0) *sbad = 0;
        for (int r = tid; r < NPV; r += NT) face[r] = 0;
        __syncthreads();
        for (int i = tid; i < NPV * NPV; i += NT) sM[i] = P.M[(size_t)e * NPV * NPV + i];
        for (int i = tid; i < NPV * NPV * ND; i += NT) sMi[i] = C[i];
        for (int i = tid; i < NPV * NDF * ND; i += NT) {
            const double v = P.E[(size_t)e * NPV * NDF * ND + i];
            sMiE[i] = v;
            if (v != 0.0) face[i % NPV] = 1;             // a node of some face
        }
        for (int i = tid; i < NPV * NCU * ND; i += NT) sMiRq[i] = P.Rq[(size_t)e * NPV * NCU * ND + i];
        for (int r = tid; r < NPV; r += NT) sMi[NPV * NX + r] = probe_rhs(r);
        __syncthreads();
        // the elimination order of the local system: face nodes first, the density of each kind last
        for (int r = tid; r < NPV; r += NT) {
            int nface = 0, before = 0;
            for (int s = 0; s < NPV; s++) {
                nface += face[s];
                before += s < r && face[s] == face[r];
            }
            int *o = ord + (face[r] ? 0 : NCU * nface);
            const int n = face[r] ? nface : NPV - nface;
            o[2 * before] = r + NPV;
            o[2 * before + 1] = r + 2 * NPV;
            for (int c = 3; c < NCU; c++) o[(c - 1) * n + before] = r + NPV * c;
            o[(NCU - 1) * n + before] = r;
        }
        if (pivot_m) gj_regs<NPV, NX, NT, 8, true>(sM, sMi, fall, fall + 2 * NPV, var, slot, sbad);
        else block_gj<NPV, NX + 1, NPV, NT>(sM, sMi, pub, sbad, NaturalOrder{});
        if (!pivot_m && (!probe_ok<NPV, NT>(sM, sMi + NPV * NX, red) || *sbad)) {
            pivot_m = true;
            __syncthreads();
            goto element;
        }
        if (tid == 0 && *sbad) *sbad = 1;
        __syncthreads();
        const int bad_m = *sbad;
        // SD, the right-hand sides; G' and H - GK_q Mi E
        int next = coupled_product<ND, NPV, NCU, NDF, NU, NT>(
            0, BD + (size_t)NU * NU, sMi,
            [&](int b, int col, int r, double &sign) {
                sign = col < NPV ? 1.0 : (col < NPV + NDF ? -1.0 : 0.0);
                return col < NPV ? BD + r + NU * (col + NPV * b) : F + r + NU * (b + NCU * (col < NPV + NDF ? col - NPV : 0));
            },
            [&](int b, int col, int r, double v) {
                if (col < NPV) sSD[r + NU * (col + NPV * b)] = v;
                else if (col < NPV + NDF) sR[r + LDR * (1 + b + NCU * (col - NPV))] = v;
                else partu[r + NU * b] = v;
            });
        coupled_product<ND, NPV, NCU, NDF, NH, NT>(
            next, GK + (size_t)NH * NU, sMi,
            [&](int b, int col, int r, double &sign) {
                sign = col < NPV ? 1.0 : (col < NPV + NDF ? -1.0 : 0.0);
                return col < NPV ? GK + r + NH * (col + NPV * b) : H + r + NH * (b + NCU * (col < NPV + NDF ? col - NPV : 0));
            },
            [&](int b, int col, int r, double v) {
                if (col < NPV) sG[SG * (col + NPV * b) + r] = v;
                else if (col < NPV + NDF) ah[r + NH * (b + NCU * (col - NPV))] = -v;
                else part[r + NH * b] = v;
            });
        __syncthreads();
        for (int r = tid; r < NU; r += NT) {
            double v = P.Ru[(size_t)e * NU + r];
#pragma unroll
            for (int b = 0; b < NCU; b++) v -= partu[r + NU * b];
            sR[r] = v;
            sR[LDR * (1 + NH) + r] = probe_rhs(r);
        }
        __syncthreads();
        if (pivot_sd) {
            gj_regs<NU, 1 + NH, NT, 8, true, LDR>(sSD, sR, fall, fall + 2 * NU, var, slot, sbad);
        } else {
            block_gj<NU, 2 + NH, LDR, NT>(sSD, sR, pub, sbad, TableOrder{ord});
            if (!probe_ok<NU, NT>(sSD, sR + LDR * (1 + NH), red) || *sbad != bad_m) {
                pivot_sd = true;
                ah = dd;                                 // AE may lie over H: it keeps what it has (dd is written below)
                __syncthreads();
                goto element;
            }
        }
        if (tid == 0 && *sbad && !bad_m) *sbad = 2;
        // DUDG = [du, Mi Rq + Mi C du] and FE = Rh - GK_q Mi Rq - G' du
        for (int i = tid; i < NQ; i += NT) {
            const int r = i % NPV, c = i / NPV;
            double v;
            if (c < NCU) {
                v = sR[r + NPV * c];
            } else {
                const int a = (c - NCU) % NCU, d = (c - NCU) / NCU;
                v = sMiRq[r + NPV * (a + NCU * d)];
#pragma unroll
                for (int s = 0; s < NPV; s++) v += sMi[r + NPV * (s + NPV * d)] * sR[s + NPV * a];
            }
            P.DUDG[(size_t)e * NQ + i] = v;
        }
        for (int i = tid; i < (4 * NH + 31) / 32 * 32; i += NT) {
            const int r = i >> 2;
            double v = 0.0;
            if (r < NH)
                for (int k = i & 3; k < NU; k += 4) v += sG[SG * k + r] * sR[k];
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (r < NH && (i & 3) == 0) {
#pragma unroll
                for (int b = 0; b < NCU; b++) v += part[r + NH * b];
                P.FE[(size_t)e * NH + r] = P.Rh[(size_t)e * NH + r] - v;
            }
        }
        // DUDG_DUH, and AE += G' dlu in jobs of 8 columns by TO tiles of 8 rows
        for (int k = w; k < NH; k += NT / 32)
            for (int r = lane; r < NU; r += 32) store_out(dd + (size_t)NQ * k + r, sR[LDR * (1 + k) + r]);
        q_rows<NPV, ND, NCU, NDF, NH, LDR, NQ, NT>(sR + LDR, sMi, sMiE, dd + NU, wide);
        constexpr int OT = (NH + 7) / 8, TO = OT % 5 == 0 ? 5 : (OT % 4 == 0 ? 4 : (OT % 3 == 0 ? 3 : 2)), GO = (OT + TO - 1) / TO;
        for (int job = w; job < OT * GO; job += NT / 32) {
            const int c0 = 8 * (job % OT) + m, o0 = 8 * TO * (job / OT);
            const bool in = NH % 8 == 0 || c0 < NH;
            const int c = in ? c0 : NH - 1;
            double acc[TO][2], ini[TO][2];
#pragma unroll
            for (int t = 0; t < TO; t++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int o = o0 + 8 * t + 2 * q + h;
                    ini[t][h] = ae[NH * c + (o < NH ? o : NH - 1)];
                    acc[t][h] = 0.0;
                }
#pragma unroll 4
            for (int s = 0; s < (NU + 3) / 4; s++) {
                const bool ink = NU % 4 == 0 || 4 * s + q < NU;
                const int k = ink ? 4 * s + q : NU - 1;
                double l = sR[LDR * (1 + c) + k];
                if constexpr (NU % 4 != 0) l = ink ? l : 0.0;
#pragma unroll
                for (int t = 0; t < TO; t++) {
                    const int o = o0 + 8 * t + m;
                    double g = sG[SG * k + (o < NH ? o : NH - 1)];
                    if constexpr (NU % 4 != 0) g = ink ? g : 0.0;
                    dmma(acc[t], l, g);
                }
            }
            if (in) {
#pragma unroll
                for (int t = 0; t < TO; t++) {
                    const int o = o0 + 8 * t + 2 * q;
                    if (o + 1 < NH) store2(ae + NH * c + o, acc[t][0] + ini[t][0], acc[t][1] + ini[t][1], wide && NH % 2 == 0);
                    else if (o < NH) store_out(ae + NH * c + o, acc[t][0] + ini[t][0]);
                }
            }
        }
        if (tid == 0 && P.status) P.status[e] = *sbad;
        __syncthreads();
    }
}

}  // namespace hdgx
