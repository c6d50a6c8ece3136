// factor_level.cu -- one colour or level of the block ILU(0) factorisation (kernel/computeBILU0.m:11-46),
// one CTA per row, for the block sizes of the element shapes and rows of at most 6 neighbours.
//
// For the neighbours k of row i that are eliminated before it, in their order:
//   L = A_ik inv(U_kk);  A_ik <- L;  A_ij <- A_ij - L U_kj   (j = i or a neighbour of both, after k)
// then A_ii <- inv(A_ii).  The products run on FP64 tensor-core fragments out of shared memory, the
// inverse by block_gj (checked in every column, and repeated with partial pivoting when the check fails).
//
// What bounded the factorisation was the length of one row's chain, once per level: index loads one
// after another in one thread, products that read both factors from L2 for every output, an inverse
// with a barrier per unknown, and a launch.  Here a warp looks up all neighbours of all neighbours
// at once; the row's own blocks, which no other row changes, are fetched while the level before
// still runs (programmatic dependent launch), and neighbour s + 1's blocks while s's are used.
// Factorisation: 2D p = 3, 12,416 faces, 440 levels: 11.4 -> 2.83 ms; 3D p = 2, 6,528 faces, 282
// levels: 37.7 -> 5.25 ms.
#include <cuda_runtime.h>
#include "dmma.cuh"
#include "hdgx_common.cuh"
#include "trace_internal.cuh"

namespace hdgx {

template <int BS>
struct FactorShape {
    static constexpr int MAXD = 6, NP = (BS + 7) / 8 * 8, LD = (NP + 4 - NP % 8 + 7) / 8 * 8 - 4;   // LD = 4 modulo 8
    // A warp or two for every tile row of a block.  Factorisation in ms with half as many / these / twice as many threads:
    // blocks of 8, 415 levels, 1.97 / 1.79 / 1.79; of 12, 272, 2.22 / 1.74 / 1.57; of 15, 515, 12.9 / 8.06 / 6.02; of 16, 440,
    // 3.31 / 2.72 / 2.58; of 20, 205, 2.25 / 1.88 / 1.64; of 30, 282, 6.58 / 5.33 / 4.69.
    static constexpr int NT = BS >= 20 ? 256 : (BS > 8 ? 128 : 64);
    static constexpr int BLK = LD * NP;                     // doubles of a block in shared memory, padded with zeros
    static constexpr int MAXT = 4, ALLT = MAXD + 1;         // blocks of row i that one neighbour changes: staged
                                                            // together (a tetrahedron's faces need 3), in all
    static constexpr int STAGE = 1 + MAXT;                  // inv(U_kk) and those U_kj
    static constexpr int o_row = 0, o_stage = o_row + (MAXD + 1) * BLK, o_T = o_stage + 2 * STAGE * BLK;
    static constexpr int o_A = o_T + BLK, o_B = o_A + BS * BS, o_pub = (o_B + BS * BS + 1) / 2 * 2;
    static constexpr int doubles = o_pub + BlockGJ<BS, 1, 32>::pub_doubles;
    // per neighbour in elimination order: its place in row i, its diagonal block, the number of targets, and
    // (place in row i, block U_kj) of each; then scratch of the pivoted inverse
    static constexpr int i_n = 0, i_at = 2, i_diag = i_at + MAXD, i_nt = i_diag + MAXD, i_tgt = i_nt + MAXD,
                         i_src = i_tgt + MAXD * ALLT, i_var = i_src + MAXD * ALLT, i_slot = i_var + BS, i_bad = i_slot + 2,
                         ints = i_bad + 2;
    static constexpr size_t bytes = sizeof(double) * doubles + sizeof(int) * ints;
    static_assert(bytes <= 227 * 1024, "a row fits shared memory");
};

// What the check of an inverse (inverse_ok, every column) allows; beyond, it is done again with pivoting.  Over
// 138,000 diagonal blocks of 2D and 3D, Euler and NS, all sizes, the elimination leaves at most 1.3e-15, in 9 of 10
// at most 3.2e-16; with a pivot pair of determinant d (the block of order 1) it leaves some 1e-16 / d.
constexpr double kInverseError = 4e-15;

// 16 bytes from L2 (never from L1, which could hold what another level's kernel has changed since)
__device__ __forceinline__ void copy_async16(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

template <int BS>
__global__ void __launch_bounds__(FactorShape<BS>::NT)
    bilu0_row_kernel(const int *__restrict__ rows, int nrows, const long long *__restrict__ rowpts,
                     const int *__restrict__ colind, const int *__restrict__ pos, double *Mg, int *status) {
    using S = FactorShape<BS>;
    constexpr int NT = S::NT, NW = NT / 32, LD = S::LD, BLK = S::BLK, MAXD = S::MAXD, MAXT = S::MAXT, ALLT = S::ALLT, B2 = BS * BS,
                  TN = S::NP / 8;
    extern __shared__ __align__(16) double sm[];
    double *row = sm + S::o_row, *stage = sm + S::o_stage, *T = sm + S::o_T, *A = sm + S::o_A, *B = sm + S::o_B;
    int *si = reinterpret_cast<int *>(sm + S::doubles);
    int *s_n = si + S::i_n, *s_at = si + S::i_at, *s_diag = si + S::i_diag, *s_nt = si + S::i_nt, *s_tgt = si + S::i_tgt,
        *s_src = si + S::i_src, *s_bad = si + S::i_bad;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, m = lane >> 2, q = lane & 3;
    const unsigned full = 0xffffffffu;
    // the level after this one may begin with what does not depend on it
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (S::NP > BS) {                                       // the padding of the blocks: zeros, once
        for (int t = tid; t < S::o_A; t += NT) sm[t] = 0.0;
        __syncthreads();
    }
    // block `from` of Mg into shared memory (leading dimension LD)
    const bool wide = BS % 2 == 0 && ((size_t)Mg & 15) == 0;
    auto fetch = [&](double *to, long long from) {
        const double *src = Mg + (size_t)B2 * from;
        if (wide) {
            for (int t = 2 * tid; t < B2; t += 2 * NT) copy_async16(to + t % BS + LD * (t / BS), src + t);
        } else {
            for (int t = tid; t < B2; t += NT) to[t % BS + LD * (t / BS)] = __ldcg(src + t);
        }
    };
    // C = A B or C -= A B, tiles of 8 x 8 over the warps from tile t0 of the CTA's round on
    auto product = [&](double *Cm, const double *Am, const double *Bm, bool subtract, int t0) {
        for (int t = (w + NW - t0 % NW) % NW; t < TN * TN; t += NW) {
            const int r0 = 8 * (t % TN), c0 = 8 * (t / TN);
            double acc[2] = {0.0, 0.0};
#pragma unroll
            for (int s = 0; s < S::NP / 4; s++) dmma(acc, Am[r0 + m + LD * (4 * s + q)], Bm[4 * s + q + LD * (c0 + m)]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                // the padding stays zero: what a singular block puts there would reach the CTA's next row
                if (BS % 8 != 0 && (r0 + m >= BS || c0 + 2 * q + h >= BS)) continue;
                double *c = Cm + r0 + m + LD * (c0 + 2 * q + h);
                *c = subtract ? *c - acc[h] : acc[h];
            }
        }
    };
    bool waited = false;
    for (int qi = blockIdx.x; qi < nrows; qi += gridDim.x) {
        const int i = rows[qi];
        const long long k0 = rowpts[i];
        const int deg = min((int)(rowpts[i + 1] - k0) - 1, MAXD);
        fetch(row, k0);
        for (int d = 0; d < deg; d++) fetch(row + (1 + d) * BLK, k0 + 1 + d);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (w == 0) {
            const int j = lane < deg ? colind[k0 + 1 + lane] - 1 : -1;
            const int pi = pos[i], pj = j >= 0 ? pos[j] : 0;
            const bool before = j >= 0 && pj < pi;
            const int n = __popc(__ballot_sync(full, before));
            int rank = 0;
            for (int t = 0; t < deg; t++) {
                const int pt = __shfl_sync(full, pj, t), bt = __shfl_sync(full, (int)before, t);
                rank += bt && pt < pj;
            }
            const long long r0 = j >= 0 ? rowpts[j] : 0;
            const int dj = j >= 0 ? (int)(rowpts[j + 1] - r0) - 1 : 0;
            if (before) {
                s_at[rank] = lane;
                s_diag[rank] = (int)r0;
            }
            // lane t runs through the row of neighbour t; its blocks U_tj with j = i or a neighbour of i after t
            int nt = 0;
            for (int u = 0; u < MAXD; u++) {
                const int c = before && u < dj ? colind[r0 + 1 + u] - 1 : -2;
                int target = c == i ? 0 : -1;
                bool after = c == i;
                for (int t = 0; t < deg; t++) {
                    const int jt = __shfl_sync(full, j, t), pt = __shfl_sync(full, pj, t);
                    if (c == jt) {
                        target = 1 + t;
                        after = pt > pj;
                    }
                }
                if (before && target >= 0 && after && nt < ALLT) {
                    s_tgt[rank * ALLT + nt] = target;
                    s_src[rank * ALLT + nt] = (int)(r0 + 1 + u);
                    nt++;
                }
            }
            if (before) s_nt[rank] = nt;
            if (lane == 0) {
                *s_n = n;
                *s_bad = 0;
            }
        }
        if (!waited) {                                       // the levels before are complete from here on
            asm volatile("griddepcontrol.wait;" ::: "memory");
            waited = true;
        }
        __syncthreads();
        const int n = *s_n;
        auto stage_row = [&](int s) {
            double *to = stage + (s & 1) * S::STAGE * BLK;
            if (s < n) {
                fetch(to, s_diag[s]);
                for (int t = 0; t < min(s_nt[s], MAXT); t++) fetch(to + (1 + t) * BLK, s_src[s * ALLT + t]);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        stage_row(0);
        for (int s = 0; s < n; s++) {
            stage_row(s + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            double *from = stage + (s & 1) * S::STAGE * BLK;
            double *Aik = row + (1 + s_at[s]) * BLK;
            product(T, Aik, from, false, 0);
            __syncthreads();
            for (int t = 0; t < min(s_nt[s], MAXT); t++)
                product(row + s_tgt[s * ALLT + t] * BLK, T, from + (1 + t) * BLK, true, t * TN * TN);
            for (int t = MAXT; t < s_nt[s]; t++) {           // more common neighbours than a mesh of simplices has
                __syncthreads();
                fetch(from + BLK, s_src[s * ALLT + t]);
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();
                product(row + s_tgt[s * ALLT + t] * BLK, T, from + BLK, true, 0);
            }
            for (int t = tid; t < B2; t += NT) {
                const int at = t % BS + LD * (t / BS);
                Mg[(size_t)B2 * (k0 + 1 + s_at[s]) + t] = T[at];
            }
            __syncthreads();
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // the blocks of the neighbours after i as they are now; inv(A_ii)
        for (int d = 0; d < deg; d++) {
            bool lower = false;
            for (int s = 0; s < n; s++) lower |= s_at[s] == d;
            if (lower || n == 0) continue;
            for (int t = tid; t < B2; t += NT) Mg[(size_t)B2 * (k0 + 1 + d) + t] = row[(1 + d) * BLK + t % BS + LD * (t / BS)];
        }
        for (int t = tid; t < B2; t += NT) {
            A[t] = row[t % BS + LD * (t / BS)];
            B[t] = t % BS == t / BS ? 1.0 : 0.0;
        }
        __syncthreads();
        block_gj<BS, BS, BS, NT>(A, B, sm + S::o_pub, s_bad, NaturalOrder{});
        const bool ok = inverse_ok<BS, NT>(A, B, kInverseError);
        if (!ok || *s_bad) {
            __syncthreads();
            if (tid == 0) *s_bad = 0;
            __syncthreads();
            double *f = sm + S::o_pub;
            gj_regs_t<double, BS, 0, BS, true, NT, 8, true>(A, nullptr, B, f, f + 2 * BS, si + S::i_var, si + S::i_slot, s_bad);
        }
        for (int t = tid; t < B2; t += NT) Mg[(size_t)B2 * k0 + t] = B[t];
        if (tid == 0 && *s_bad && status) status[i] = 1;
        __syncthreads();
    }
}

template <int BS>
static int launch_rows(const hdgx_bsr *A, const int *rows, int nr, double *Mg, int *status, bool first, cudaStream_t st) {
    using S = FactorShape<BS>;
    auto kern = bilu0_row_kernel<BS>;
    if (allow_dynamic_smem((const void *)kern, S::bytes) != cudaSuccess) return -10;
    cudaLaunchConfig_t cfg = {};
    const int cap = sm_count_of(current_device()) * 4;
    cfg.gridDim = dim3(nr < cap ? nr : cap);
    cfg.blockDim = dim3(S::NT);
    cfg.dynamicSmemBytes = S::bytes;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = first ? 0 : 1;       // the first level waits for all work before it
    return cudaLaunchKernelEx(&cfg, kern, rows, nr, (const long long *)A->rowpts, (const int *)A->colind, (const int *)A->pos, Mg,
                              status) == cudaSuccess
               ? 0
               : -12;
}

// The rows of one level; first: the factorisation's first launch.  0 launched, 1 no specialisation (the
// caller runs the general kernel), negative: failed.  A sweep plan says that no row has more than
// sweep_maxd neighbours.
int factor_level(const hdgx_bsr *A, const int *rows, int nr, double *Mg, int *status, bool first, cudaStream_t st) {
    if (!A->sweep_plan || (A->sweep_maxd != 4 && A->sweep_maxd != 6)) return 1;
    switch (A->bs) {
#define HDGX_FR(B) case B: return launch_rows<B>(A, rows, nr, Mg, status, first, st);
        HDGX_FR(8) HDGX_FR(12) HDGX_FR(15) HDGX_FR(16) HDGX_FR(20) HDGX_FR(30)
#undef HDGX_FR
        default: return 1;
    }
}

}  // namespace hdgx
