// level_sweep.cu -- BILU(0) application (kernel/applyBILU0.m:10-48) as ONE data-driven launch.
//
// A sequential elimination order such as the minimum-discarded-fill order of
// kernel/computeMDFordering.m has long dependency chains: on the 2D NS p = 3 mesh of 49,408
// faces the level schedule has 1,100 levels of 45 rows on average, and the apply is bound by
// the latency of a level, not by the 0.5 GB of factors it reads.  Here a warp owns a row, and a
// row starts when the values it needs have arrived, not when a whole level is done.
//
// Work split: slot q of the plan (rows in level order) belongs to warp q % W of a grid of W warps
// that are resident together (one cluster, or a cooperative launch).  A warp walks its slots in
// ascending order in the forward sweep and in descending order in the backward sweep:
//   y_i = x_i - sum_j L_ij y_j                   (rows j eliminated before i)
//   v_i = inv(U_ii) (y_i - sum_j U_ij v_j)       (rows j eliminated after i; inverses are stored)
// The row with the lowest unfinished slot never waits, so the sweep always advances.
//
// A value is its own ready flag: y and v are filled with kPending (all bits set, a NaN no kernel
// here produces: a result with these bits is stored as the default NaN) before the launch, and a
// reader polls the value itself at L2 until it differs.  One store and one load carry a row to its
// readers; there is no fence, no barrier and no separate flag.  Waits are bounded (kPollLimit
// polls, then NaN is used and passed on and *err, where there is one, is set, so that a plan that
// is not a schedule ends in NaN and in an error of the solve, never in a hang).
//
// What bounds a level is then the store-to-load time through L2 (0.47 us measured between two SMs)
// and the arithmetic after it, so both are kept short: the row's factor blocks are staged in
// shared memory before its inputs arrive, by one bulk copy a block (copies of single values by all lanes cost a
// warp about 2,500 cycles a row of 30 x 30 blocks; blocks that are no multiple of 16 bytes, those of 15 x 15, and
// factors that are not aligned to 16 still take them: apply, with four warps a row of an average level, 600 -> 577 us
// at 12,416 faces of 16, 597 -> 567 us at 6,528 of 30), lane r of part p (PARTS = 32 / BS parts) adds up only
// the neighbours p, p + PARTS, .. in CH independent chains (a dependent FP64 multiply-add takes
// 17.6 cycles), and the parts are added with shuffles.  Apply: 571 us at those faces of 16, 539 us at those of 30.
#include <cuda_runtime.h>
#include <type_traits>
#include "hdgx_common.cuh"
#include "trace_internal.cuh"

namespace hdgx {

cudaMemPool_t device_pool();             // the library's pool of the current device (solve.cu)

constexpr unsigned long long kPending = ~0ull;
constexpr int kPollLimit = 1 << 21;

__device__ __forceinline__ void bulk_prefetch_l2(const void *p, unsigned bytes) {
    // the 16-byte aligned interior of [p, p + bytes) (a bulk prefetch needs aligned ends)
    const unsigned long long a0 = ((unsigned long long)p + 15) & ~15ull;
    const unsigned long long a1 = ((unsigned long long)p + bytes) & ~15ull;
    if (a1 > a0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a0), "r"((unsigned)(a1 - a0)) : "memory");
}
__device__ __forceinline__ unsigned long long load_value(const double *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_value(double *p, double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (b == kPending) b = 0x7ff8000000000000ull;
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
// One warp's mbarrier for its bulk copies
__device__ __forceinline__ void stage_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void stage_bulk(void *dst, const void *src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool stage_wait(unsigned bar, unsigned parity, int limit) {
    unsigned done = 0;
    for (int n = 0; !done && n < limit; n++)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(bar), "r"(parity)
                     : "memory");
    return done;
}

// Shared memory of one warp: MAXD neighbour blocks and the diagonal block of its row, the
// neighbours' values, the row's intermediate t and the mbarrier; as many warps per CTA as fit (at most 16).
template <int BS, int MAXD, class MT>
struct SweepShape {
    static constexpr int PARTS = 32 / BS, DP = (MAXD + PARTS - 1) / PARTS;
    static constexpr int RW = 2 + 4 * MAXD;                                  // record width (ints)
    static constexpr int BLK = BS * BS;
    // Chains of a row's sum: enough that the multiply-adds' latency is hidden, few enough that adding them up is
    // short.  Apply in us with half as many / these / twice as many: blocks of 8, 10,920 faces, 472 / 433 / 435; of 12,
    // 4,880, 301 / 301 / 312; of 15, 12,600, 957 / 963 / 974; of 16, 12,416, 593 / 571 / 581; of 20, 2,760, 307 / 306 / 323;
    // of 30, 6,528, 549 / 542 / 544.
    static constexpr int CH = BS == 30 ? 6 : (BS == 15 ? 5 : 4);
    static constexpr size_t stage = (sizeof(MT) * BLK * (MAXD + 1) + 15) / 16 * 16;
    static constexpr int BSP = (BS + 1) / 2 * 2;                             // 16-byte aligned value rows
    static constexpr size_t warp_bytes = stage + sizeof(double) * BSP * (MAXD + 1) + 16;
    static constexpr int fit = (int)(216 * 1024 / warp_bytes);
    static constexpr int WPC = fit > 16 ? 16 : fit;
    static constexpr size_t smem = warp_bytes * WPC;
    // Products of the neighbours that have arrived, while the last one is waited for: pays where a block's product
    // is long.  Apply in us, all at once / as they arrive (four warps a row, values copied one by one): blocks of 30, 6,528
    // faces in 282 levels, 702 / 597; of 20, 1,776 in 160, 251 / 255; of 16, 12,416 in 440, 592 / 623; of 12, 800 in 104, 129 / 133.
    // Each product has a sum of its own, and these are added in slot order, so that the result does not depend on who
    // came first (one sum in the order of arrival: 536 us instead of 539; products in slot order, each when it and
    // those before it are there: 614).
    static constexpr bool EARLY = BS > 20;
    static_assert(!EARLY || (PARTS == 1 && DP <= 6), "the slots of a warp are one row's");
    static_assert(BS <= 32 && RW <= 32 && WPC >= 1, "one lane per row component and per record entry");
};

// columns [c0, c0 + N) of a row of the block at B (its first column) times the values u, added to CH chains
template <int BS, int N, int CH, class MT>
__device__ __forceinline__ void dot_cols(const MT *B, const double *u, int c0, double (&acc)[CH]) {
#pragma unroll
    for (int c = 0; c < N; c++)
        if (BS % N == 0 || c0 + c < BS) acc[c % CH] = fma((double)B[BS * (c0 + c)], u[c0 + c], acc[c % CH]);
}
template <int CH>
__device__ __forceinline__ double chain_sum(const double (&acc)[CH]) {
    double t = acc[0] + acc[1];
#pragma unroll
    for (int c = 2; c < CH; c += 2) t += c + 1 < CH ? acc[c] + acc[(c + 1) % CH] : acc[c];
    return t;
}

template <int BS, int MAXD, class MT>
__global__ void __launch_bounds__(SweepShape<BS, MAXD, MT>::WPC * 32)
    bilu0_sweep_kernel(int nf, const int *__restrict__ rec, const MT *__restrict__ Mg, const double *__restrict__ x,
                       double *y, double *v, int phases, int *err) {
    using S = SweepShape<BS, MAXD, MT>;
    constexpr int PARTS = S::PARTS, DP = S::DP, RW = S::RW, BLK = S::BLK, BSP = S::BSP, CH = S::CH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *mine = smem_raw + S::warp_bytes * warp;
    MT *blk = reinterpret_cast<MT *>(mine);                          // [MAXD + 1][BS, BS]
    double *val = reinterpret_cast<double *>(mine + S::stage);       // [MAXD][BSP], then t [BSP]
    double *tsh = val + MAXD * BSP;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(tsh + BSP);
    const int part = lane / BS, r = lane - part * BS;
    const bool on = part < PARTS;
    const int W = gridDim.x * S::WPC, w = warp * gridDim.x + blockIdx.x;   // neighbouring slots on different SMs
    const bool wide = sizeof(MT) * BLK % 16 == 0 && ((size_t)Mg & 15) == 0;   // a bulk copy's addresses and sizes
    int limit = kPollLimit, stage_limit = kPollLimit;
    unsigned parity = 0;                                             // of the row staged next
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();

    // slot record, one entry per lane: (row, diagonal block, MAXD (block, column) of the earlier
    // neighbours, MAXD of the later ones)
    auto record = [&](int q) { return (q >= 0 && q < nf && lane < RW) ? __ldg(rec + (size_t)q * RW + lane) : -1; };
    auto stage_block = [&](int slot, int k) {
        const MT *src = Mg + (size_t)BLK * k;
        MT *dst = blk + slot * BLK;
        for (int t = lane; t < BLK; t += 32) cp_async<sizeof(MT)>(dst + t, src + t);
    };
    auto add_parts = [&](double s) {
        double t = s;
#pragma unroll
        for (int p = 1; p < PARTS; p++) t += __shfl_down_sync(0xffffffffu, s, p * BS);
        return t;                                                        // valid in part 0
    };

    auto sweep = [&](auto dir) {
        constexpr bool BWD = decltype(dir)::value;
        constexpr int OFF = BWD ? 2 + 2 * MAXD : 2;
        const double *in = BWD ? v : y;
        double *out = BWD ? v : y;
        const int step = BWD ? -W : W;
        int q = BWD ? nf - 1 - w : w;
        int cur = record(q), nxt = record(q + step), nxt2 = record(q + 2 * step);
        auto begin_row = [&](int R) {                                    // stage the row's blocks
            if (__shfl_sync(0xffffffffu, R, 0) < 0) return;
            if (wide) {                                                  // lane d: block d
                const int k = __shfl_sync(0xffffffffu, R, lane < MAXD ? OFF + 2 * lane : 1);
                const bool has = (lane < MAXD || (BWD && lane == MAXD)) && k >= 0;
                const unsigned n = __popc(__ballot_sync(0xffffffffu, has));
                if (lane == 0) stage_expect(bar, n * (unsigned)(sizeof(MT) * BLK));
                __syncwarp();
                if (has) stage_bulk(blk + lane * BLK, Mg + (size_t)BLK * k, sizeof(MT) * BLK, bar);
                return;
            }
#pragma unroll
            for (int d = 0; d < MAXD; d++) {
                const int k = __shfl_sync(0xffffffffu, R, OFF + 2 * d);
                if (k >= 0) stage_block(d, k);
            }
            if (BWD) stage_block(MAXD, __shfl_sync(0xffffffffu, R, 1));
        };
        auto prefetch_row = [&](int R) {                                 // the blocks of a later row into L2
            const int at = lane < MAXD ? OFF + 2 * lane : 1;
            const int k = __shfl_sync(0xffffffffu, R, at);
            if ((lane < MAXD || (BWD && lane == MAXD)) && k >= 0) bulk_prefetch_l2(Mg + (size_t)BLK * k, sizeof(MT) * BLK);
        };
        begin_row(cur);
        prefetch_row(nxt);
        auto load_x = [&](int R) {
            const int i = __shfl_sync(0xffffffffu, R, 0);
            return (!BWD && i >= 0 && on) ? __ldg(x + (size_t)BS * i + r) : 0.0;
        };
        double xv = load_x(cur);
        while (q >= 0 && q < nf) {
            const int i = __shfl_sync(0xffffffffu, cur, 0);
            int k[DP], j[DP];
#pragma unroll
            for (int s = 0; s < DP; s++) {
                const int d = part + s * PARTS;
                const int at = OFF + 2 * (d < MAXD ? d : 0);
                k[s] = __shfl_sync(0xffffffffu, cur, at);
                j[s] = __shfl_sync(0xffffffffu, cur, at + 1);
                if (!on || d >= MAXD) k[s] = -1;
            }
            prefetch_row(nxt2);
            const int nxt3 = record(q + 3 * step);
            bool staged = true;
            if (wide) {
                staged = stage_wait(bar, parity, stage_limit);
                if (!staged) {
                    stage_limit = 1;
                    if (err && lane == 0) atomicExch(err, 1);
                }
                parity ^= 1;
            } else {
                asm volatile("cp.async.wait_all;" ::: "memory");
            }
            // wait for the neighbours' values (and, backward, for the row's own y)
            unsigned long long got[DP], own = 0;
            [[maybe_unused]] double acc[CH] = {};
            [[maybe_unused]] double each[6] = {};                        // EARLY: a neighbour's product
            unsigned todo = 0;                                           // slots whose product is to be added
#pragma unroll
            for (int s = 0; s < DP; s++) todo |= k[s] >= 0 ? 1u << s : 0u;
            auto use = [&](unsigned which) {
#pragma unroll
                for (int s = 0; s < DP; s++)
                    if (which >> s & 1) val[(part + s * PARTS) * BSP + r] = __longlong_as_double((long long)got[s]);
                __syncwarp();
#pragma unroll
                for (int s = 0; s < DP; s++) {
                    const int d = part + s * PARTS;
                    if (which >> s & 1) {
                        if constexpr (S::EARLY) {
                            double one[CH] = {};
                            dot_cols<BS, BS, CH>(blk + d * BLK + r, val + d * BSP, 0, one);
                            each[s] = chain_sum(one);
                        } else {
                            dot_cols<BS, BS, CH>(blk + d * BLK + r, val + d * BSP, 0, acc);
                        }
                    }
                }
            };
            for (int n = 0;;) {
                unsigned miss = 0;
#pragma unroll
                for (int s = 0; s < DP; s++) got[s] = todo >> s & 1 ? load_value(in + (size_t)BS * j[s] + r) : 0ull;
                if (BWD) own = part == 0 ? load_value(y + (size_t)BS * i + r) : 0ull;
#pragma unroll
                for (int s = 0; s < DP; s++) miss |= got[s] == kPending ? 1u << s : 0u;
                if (BWD) miss |= own == kPending ? 1u << DP : 0u;
                if (__all_sync(0xffffffffu, !miss)) break;
                if (++n >= limit) {                                      // NaN (kPending is one) from here on
                    limit = 1;
                    if (err && lane == 0) atomicExch(err, 1);
                    break;
                }
                if constexpr (S::EARLY) {
                    const unsigned here = __reduce_and_sync(0xffffffffu, ~miss) & todo;
                    if (__any_sync(0xffffffffu, here != 0)) {
                        use(here);
                        todo &= ~here;
                    }
                }
            }
            use(todo);
            if (!staged) xv = __longlong_as_double((long long)(own = kPending));
            double sum;
            if constexpr (S::EARLY) sum = (each[0] + each[1]) + (each[2] + each[3]) + (each[4] + each[5]);
            else sum = add_parts(chain_sum(acc));
            if (!BWD) {
                if (part == 0) store_value(out + (size_t)BS * i + r, xv - sum);
            } else {
                if (part == 0) tsh[r] = __longlong_as_double((long long)own) - sum;
                __syncwarp();
                double ad[CH] = {};
                constexpr int CP = (BS + PARTS - 1) / PARTS;             // columns of a part
                if (on) dot_cols<BS, CP, CH>(blk + MAXD * BLK + r, tsh, part * CP, ad);
                const double o = add_parts(chain_sum(ad));
                if (part == 0) store_value(out + (size_t)BS * i + r, o);
            }
            __syncwarp();                                                // the staged blocks and values are free
            cur = nxt;
            nxt = nxt2;
            nxt2 = nxt3;
            q += step;
            begin_row(cur);
            xv = load_x(cur);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    };
    if (phases & 1) sweep(std::false_type{});
    if (phases & 2) sweep(std::true_type{});
}

__global__ void fill_pending_kernel(size_t n, unsigned long long *a, unsigned long long *b) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        if (a) a[t] = kPending;
        if (b) b[t] = kPending;
    }
}

// The grid must be resident at once.  Up to 8 CTAs are one cluster, which the hardware places
// together or not at all, so that the sweeps of many concurrent solves share the GPU; larger grids
// are a cooperative launch.
template <int BS, int MAXD, class MT>
static int launch_sweep(const hdgx_bsr *A, const MT *Mg, const double *x, double *y, double *v, bool apart, int *err,
                        cudaStream_t st) {
    using S = SweepShape<BS, MAXD, MT>;
    auto kern = bilu0_sweep_kernel<BS, MAXD, MT>;
    if (allow_dynamic_smem((const void *)kern, S::smem) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    const int nf = A->nf;
    const size_t n = (size_t)BS * nf;
    // four warps per row of an average level, so that a row's warp is there, its blocks staged, when
    // the values arrive; six where a block takes long to stage.  Apply in us with 2, 3, 4 and 6 (clusters of
    // at most 8 CTAs): 2D p = 3, 12,416 faces in 440 levels, 692, 577, 577, 559; 49,408 in 888, 1,507, 1,318, 1,237 to 1,333, 1,289;
    // 3D p = 2, 6,528 faces in 282 levels, 705, 603, 567, 533.  More warps take SMs from other solves:
    // 32 queued 2D requests on 16 slots ran at 34 to 43 solves/s with four, 16 to 29 with eight.
    const long long want = ((S::EARLY ? 6ll : 4ll) * nf / A->ncolors + S::WPC - 1) / S::WPC;
    const int nsm = sm_count_of(current_device());
    int G = want < 1 ? 1 : (want > nsm ? nsm : (int)want);
    if (G <= 8) G = G > 4 ? 8 : (G > 2 ? 4 : G);
    const int *rec = A->sweep_plan + A->ncolors + 1;
    const unsigned fg = (unsigned)((n + 255) / 256 < (size_t)nsm * 8 ? (n + 255) / 256 : (size_t)nsm * 8);
    auto launch = [&](int phases) -> bool {
        if (G > 8) {
            int nf_ = nf, ph = phases;
            void *args[] = {&nf_, &rec, &Mg, &x, &y, &v, &ph, &err};
            if (cudaLaunchCooperativeKernel((const void *)kern, dim3(G), dim3(S::WPC * 32), args, S::smem, st) == cudaSuccess)
                return true;
            cudaGetLastError();
            G = 8;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(G);
        cfg.blockDim = dim3(S::WPC * 32);
        cfg.dynamicSmemBytes = S::smem;
        cfg.stream = st;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = G;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kern, nf, rec, Mg, x, y, v, phases, err) == cudaSuccess;
    };
    unsigned long long *yb = reinterpret_cast<unsigned long long *>(y), *vb = reinterpret_cast<unsigned long long *>(v);
    if (!apart) {                                       // v over x: x is read before v is marked
        fill_pending_kernel<<<fg, 256, 0, st>>>(n, yb, nullptr);
        if (!launch(1)) return 1;
        fill_pending_kernel<<<fg, 256, 0, st>>>(n, vb, nullptr);
        return launch(2) ? 0 : 1;
    }
    fill_pending_kernel<<<fg, 256, 0, st>>>(n, yb, vb);
    return launch(3) ? 0 : 1;
}

// 0 when launched, 1 when there is no plan or no specialisation for it (the caller falls back to one launch per level).
// The forward sweep's values need a place of their own: where y lies over x or v, one from the library's pool takes
// its part (one launch per level instead: 10.2 ms, not 0.58, at 12,416 faces of 16 in 440 levels).
template <class MT>
static int level_sweep_apply_t(const hdgx_bsr *A, const MT *Mg, const double *x, double *y, double *v, int *err,
                               cudaStream_t st) {
    if (!A->sweep_plan || A->ncolors < 1 || A->nf < 1) return 1;
    const int md = A->sweep_maxd, bs = A->bs;
    if ((md != 4 && md != 6) || (bs != 8 && bs != 12 && bs != 15 && bs != 16 && bs != 20 && bs != 30)) return 1;
    const size_t n = (size_t)bs * A->nf;
    auto overlap = [n](const double *a, const double *b) { return a < b + n && b < a + n; };
    double *own = nullptr;
    if (overlap(x, y) || overlap(y, v)) {
        cudaMemPool_t pool = device_pool();
        if (!pool || cudaMallocFromPoolAsync((void **)&own, sizeof(double) * n, pool, st) != cudaSuccess) {
            cudaGetLastError();
            return 1;
        }
        y = own;
    }
    const bool apart = !overlap(x, v);
    int rc = 1;
    switch (bs) {
#define HDGX_LS(B)                                                                                              \
    case B:                                                                                                     \
        rc = md == 4 ? launch_sweep<B, 4, MT>(A, Mg, x, y, v, apart, err, st)                                   \
                     : launch_sweep<B, 6, MT>(A, Mg, x, y, v, apart, err, st);                                  \
        break;
        HDGX_LS(8) HDGX_LS(12) HDGX_LS(15) HDGX_LS(16) HDGX_LS(20) HDGX_LS(30)
#undef HDGX_LS
    }
    if (own) cudaFreeAsync(own, st);
    return rc;
}

int level_sweep_apply(const hdgx_bsr *A, const double *Mg, const double *x, double *y, double *v, int *err, cudaStream_t st) {
    return level_sweep_apply_t<double>(A, Mg, x, y, v, err, st);
}
// The same sweeps with the factors stored in FP32 (the mixed-precision preconditioner)
int level_sweep_apply_f32(const hdgx_bsr *A, const float *Mg, const double *x, double *y, double *v, int *err,
                          cudaStream_t st) {
    return level_sweep_apply_t<float>(A, Mg, x, y, v, err, st);
}

}  // namespace hdgx
