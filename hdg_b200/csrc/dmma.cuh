// dmma.cuh -- FP64 tensor-core building blocks of the elemental kernels (mma.sync m8n8k4 .f64: one
// instruction is 256 multiply-adds on fragments of one or two doubles per lane; tcgen05 has no
// FP64 form).  On sm_100a it issues in 18 cycles per scheduler, the rate of 8 scalar multiply-adds
// a lane, from two operand registers instead of sixteen: what it saves are shared-memory reads and
// instructions, which bound the small dense products of one element.
//
// Fragments of lane l: A (8 x 4) element (l / 4, l % 4); B (4 x 8) element (l % 4, l / 4);
// C (8 x 8) elements (l / 4, 2 (l % 4)) and (l / 4, 2 (l % 4) + 1).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <utility>

namespace hdgx {

// f(integral_constant<int, 0>) .. f(integral_constant<int, N - 1>)
template <class F, int... K>
__device__ __forceinline__ void unroll_for_(F &&f, std::integer_sequence<int, K...>) {
    (f(std::integral_constant<int, K>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void unroll_for(F &&f) {
    unroll_for_(f, std::make_integer_sequence<int, N>{});
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// 1 / x from the hardware's approximation (rcp.approx.ftz.f64, which reads and returns the upper 32 bits of a
// double: a relative error e of some 2^-20) and one step of the third-order Newton (Householder) iteration
// y (1 + e + e^2), e = 1 - x y, which leaves e^3, below 2^-59, and two roundings: within 2 ulp of the quotient
// (compared with it in tests/test_range_gpu.py), in three dependent operations (the compiled division takes 230
// cycles in a dependent chain, this takes about 90).  For x and 1 / x that are normal numbers; see rcp_in_range.
__device__ __forceinline__ double fast_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// Whether fast_rcp holds: x and 1 / x normal numbers, with a margin (exponents -1020 to 1020; so x is a number,
// not zero and not infinite).
__device__ __forceinline__ bool rcp_in_range(double x) {
    return (unsigned)((__double2hiint(x) >> 20 & 2047) - 3) <= 2040u;
}

// Inverse of the 8 x 8 matrix held as a C fragment by a warp, in place: Gauss-Jordan over the four
// diagonal 2 x 2 blocks in order (no pivoting).  One 2 x 2 block costs one shuffle round, one
// reciprocal (of its determinant, the products with it formed meanwhile) and two multiply-adds in
// sequence; between(b) is issued while block b's reciprocal is on its way.  Returns false when a
// determinant is zero, not finite or outside the range of fast_rcp.
template <class F>
__device__ __forceinline__ bool inv8(double (&z)[2], F between) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, m = lane >> 2, h = lane & 3;
    bool ok = true;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const int p = 2 * b, row0 = 4 * p + b, row1 = row0 + 4;          // lanes that hold the 2 x 2 block
        const double a00 = __shfl_sync(full, z[0], row0), a01 = __shfl_sync(full, z[1], row0);
        const double a10 = __shfl_sync(full, z[0], row1), a11 = __shfl_sync(full, z[1], row1);
        const double x0 = __shfl_sync(full, z[0], 4 * m + b), x1 = __shfl_sync(full, z[1], 4 * m + b);
        const double r00 = __shfl_sync(full, z[0], 4 * p + h), r01 = __shfl_sync(full, z[1], 4 * p + h);
        const double r10 = __shfl_sync(full, z[0], 4 * p + 4 + h), r11 = __shfl_sync(full, z[1], 4 * p + 4 + h);
        const double det = fma(a00, a11, -(a01 * a10));
        ok &= rcp_in_range(det);
        const double rd = fast_rcp(det);
        between(b);
        // the block's rows become its inverse times them; row m loses (x0, x1) inverse times them
        const bool in0 = m == p, in1 = m == p + 1;
        const double u0 = in0 ? -a11 : (in1 ? a10 : fma(x0, a11, -(x1 * a10)));
        const double u1 = in0 ? a01 : (in1 ? -a00 : fma(x1, a00, -(x0 * a01)));
        const double w0 = u0 * rd, w1 = u1 * rd;
        const bool inside = in0 || in1;
        if (h == b) {
            z[0] = -w0;
            z[1] = -w1;
        } else {
            z[0] = fma(-w1, r10, fma(-w0, r00, inside ? 0.0 : z[0]));
            z[1] = fma(-w1, r11, fma(-w0, r01, inside ? 0.0 : z[1]));
        }
    }
    return ok;
}

// Elimination orders: position i of the order -> row of the system.
struct NaturalOrder {
    __device__ __forceinline__ int operator()(int i) const { return i; }
};
struct TableOrder {
    const int *at;
    __device__ __forceinline__ int operator()(int i) const { return at[i]; }
};

// Block Gauss-Jordan elimination of [A | B] (A: N x N, B: N x NR, column-major, leading dimensions N
// and LDB) without pivoting, in the order Order, B overwritten by the solution, A left as it is; by all NT
// threads.
//
// The transposed system lives in C fragments: warp w holds the columns 8 c .. 8 c + 7 of [A | B] for
// c = w, w + NT / 32, .., as tiles Z(c, i)(m, n) = [A | B](8 i + n, 8 c + m).  A block step k makes
//   Z(c, k) <- Z(c, k) inv(D)^T,   Z(c, i) <- Z(c, i) - Z(c, k) L(i)^T   (i != k)
// with D = A(k, k) and L(i) = A(i, k): the left factor is a tile the warp holds, and a C fragment is
// an A fragment of the columns 2 (l % 4) + s in step s, so no value is exchanged between lanes; the
// right factors are the 8 columns of block k, which their owner has left in shared memory (inv(D)^T
// and -L(i)^T; rows of ten doubles, so that the fragment reads are free of bank conflicts).  While
// the others update, the owner of block k + 1 brings that block up to date and inverts the next diagonal
// tile; its other columns wait until the next step (the published tiles go round three buffers), so
// that an inversion and one barrier per 8 unknowns are all that is in sequence.
// What bounds it: the chain of N / 8 inversions (about 1,300 cycles each), with the tensor work of
// other resident elements beside it.  Measured in a loop, cycles per system against an elimination
// of one unknown at a time in registers with a barrier each: N = 40, 49 right-hand sides, three
// CTAs of 192 threads per SM: 31,500 -> 14,200; N = 60, 61, one CTA of 256: 50,200 -> 19,700; N = 50,
// 121, one of 256: 45,700 -> 21,100; N = 24, 37, four of 128: 14,700 -> 6,500.
// pub: pub_doubles doubles of shared memory, 16-byte aligned, that overlap neither A nor B.
// *bad = 8 k + 1 when block k is singular, or its determinants are out of the range of fast_rcp.
// SCALED: the system is solved as (s A) x = s B with s the power of two that brings the first entry of A to 1 .. 2
// (exact, so the bits do not change), for matrices whose entries are of one size but may be very small or large (mass
// matrices: of the order of the volume): their 2 x 2 determinants leave the range first.
template <int N, int NR, int NT>
struct BlockGJ {
    static constexpr int MT = (N + 7) / 8, RT = (NR + 7) / 8, CT = MT + RT, NW = NT / 32, CPT = (CT + NW - 1) / NW;
    static constexpr int TS = 80, pub_doubles = 3 * MT * TS;
};

// Block step k on one column block, with the tiles published at `from`
template <int k, int MT>
__device__ __forceinline__ void apply_step(double (&z)[MT][2], const double *from) {
    constexpr int TS = 80;
    const int lane = threadIdx.x & 31;
    from += 20 * (lane & 3) + (lane >> 2);                      // element (row 2 (l % 4) + t, column l / 4)
    double p[2] = {0.0, 0.0};
    dmma(p, z[k][0], from[k * TS]);
    dmma(p, z[k][1], from[k * TS + 10]);
    z[k][0] = p[0];
    z[k][1] = p[1];
#pragma unroll
    for (int i = 0; i < MT; i++)
        if (i != k) {
            dmma(z[i], p[0], from[i * TS]);
            dmma(z[i], p[1], from[i * TS + 10]);
        }
}

// The owner of column block k: block step k - 1 on its tiles, the diagonal one first, then the inverse
// of the diagonal tile and the other tiles, negated, into the MT tiles at `to`.  The other tiles'
// products are issued in the gaps of the inversion.
template <int k, int MT>
__device__ __forceinline__ void publish_tiles(double (&z)[MT][2], const double *from, double *to, int *bad) {
    constexpr int TS = 80, k0 = k > 0 ? k - 1 : 0;
    const int lane = threadIdx.x & 31;
    to += 10 * (lane >> 2) + 2 * (lane & 3);
    from += 20 * (lane & 3) + (lane >> 2);
    double p[2] = {0.0, 0.0};
    auto update = [&](int i) {
        dmma(z[i], p[0], from[i * TS]);
        dmma(z[i], p[1], from[i * TS + 10]);
    };
    if constexpr (k > 0) {
        dmma(p, z[k0][0], from[k0 * TS]);
        dmma(p, z[k0][1], from[k0 * TS + 10]);
        z[k0][0] = p[0];
        z[k0][1] = p[1];
        update(k);
    }
    const bool ok = inv8(z[k], [&](int b) {
        if constexpr (k > 0) {
#pragma unroll
            for (int i = 0; i < MT; i++)
                if (i % 4 == b && i != k && i != k0) update(i);
        }
    });
    if (!ok && lane == 0 && *bad == 0) *bad = 8 * k + 1;
#pragma unroll
    for (int i = 0; i < MT; i++)
        *reinterpret_cast<double2 *>(to + i * TS) =
            i == k ? make_double2(z[i][0], z[i][1]) : make_double2(-z[i][0], -z[i][1]);
}

__device__ __forceinline__ double power_of_two_to_one(double x) {     // 2^-exponent(x); 1 when that is no normal number
    const int e = __double2hiint(x) >> 20 & 2047;
    return e >= 1 && e <= 2045 ? __hiloint2double((2046 - e) << 20, 0) : 1.0;
}

template <int N, int NR, int LDB, int NT, bool SCALED = false, class Order>
__device__ __forceinline__ void block_gj(const double *__restrict__ A, double *B, double *pub, int *bad, Order order) {
    using G = BlockGJ<N, NR, NT>;
    constexpr int MT = G::MT, CT = G::CT, NW = G::NW, CPT = G::CPT, TS = G::TS;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m = lane >> 2, n0 = 2 * (lane & 3);
    double z[CPT][MT][2];
    [[maybe_unused]] const double scale = SCALED ? power_of_two_to_one(A[0]) : 1.0;
#pragma unroll
    for (int s = 0; s < CPT; s++) {
        const int c = w + s * NW, col = 8 * c + m;
        const double *src = c < MT ? A + N * order(col < N ? col : 0) : B + LDB * (col - 8 * MT < NR ? col - 8 * MT : 0);
        const bool in = c < MT ? col < N : (c < CT && col - 8 * MT < NR);
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const int row = 8 * i + n0 + t;
                z[s][i][t] = (in && row < N) ? (SCALED ? scale * src[order(row)] : src[order(row)]) : (c < MT && col == row ? 1.0 : 0.0);
            }
    }
    auto step = [&](auto kc) {
        constexpr int k = decltype(kc)::value, kn = k + 1 < MT ? k + 1 : k, kp = k > 0 ? k - 1 : 0;
        const double *from = pub + k % 3 * MT * TS;
        auto others = [&](auto jc, int except) {                // step j on the warp's live columns but one slot
            constexpr int j = decltype(jc)::value;
#pragma unroll
            for (int s = 0; s < CPT; s++) {
                const int c = w + s * NW;
                if (c < CT && c > j && s != except) apply_step<j, MT>(z[s], pub + j % 3 * MT * TS);
            }
        };
        if (k > 0 && w == k % NW) others(std::integral_constant<int, kp>{}, k / NW);   // what it put off as publisher
        if (k + 1 < MT && w == kn % NW) publish_tiles<kn, MT>(z[kn / NW], from, pub + kn % 3 * MT * TS, bad);
        else others(std::integral_constant<int, k>{}, -1);
        __syncthreads();
    };
    if (w == 0) publish_tiles<0, MT>(z[0], pub, pub, bad);
    __syncthreads();
    unroll_for<MT>(step);
#pragma unroll
    for (int s = 0; s < CPT; s++) {
        const int c = w + s * NW, col = 8 * (c - MT) + m;
        if (c >= MT && c < CT && col < NR) {
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const int row = 8 * i + n0 + t;
                    if (row < N) B[order(row) + LDB * col] = z[s][i][t];
                }
        }
    }
    __syncthreads();
}

// The same elimination in two phases, for systems whose fragments do not fit the registers at once
// (3D p = 3: 100 unknowns, 201 right-hand sides).  block_gj_factor runs the steps on A alone and keeps
// what every step published (MT * MT tiles in `steps`, outside A); block_gj_apply then takes the right-hand
// sides through them, each warp its own 8 columns at a time, without a barrier.
template <int N, int NT, class Order>
__device__ __forceinline__ void block_gj_factor(const double *A, double *steps, int *bad, Order order) {
    constexpr int MT = (N + 7) / 8, NW = NT / 32, TS = 80;
    static_assert(MT <= NW, "one column block per warp");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m = lane >> 2, n0 = 2 * (lane & 3);
    double z[MT][2];
    const int col = 8 * w + m;
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int row = 8 * i + n0 + t;
            z[i][t] = (w < MT && col < N && row < N) ? A[order(row) + N * order(col)] : (col == row ? 1.0 : 0.0);
        }
    unroll_for<MT>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        if (w == k) publish_tiles<k, MT>(z, steps + (k - 1) * MT * TS, steps + k * MT * TS, bad);
        __syncthreads();
        if (w > k + 1 && w < MT) apply_step<k, MT>(z, steps + k * MT * TS);
    });
}

template <int N, int NR, int LDB, int NT, class Order>
__device__ __forceinline__ void block_gj_apply(double *B, const double *steps, Order order) {
    constexpr int MT = (N + 7) / 8, NW = NT / 32, TS = 80;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m = lane >> 2, n0 = 2 * (lane & 3);
    int at[MT][2];                                              // this lane's rows
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int t = 0; t < 2; t++) at[i][t] = 8 * i + n0 + t < N ? order(8 * i + n0 + t) : 0;
    for (int c = w; c < (NR + 7) / 8; c += NW) {
        const int col = 8 * c + m;
        double z[MT][2];
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const int row = 8 * i + n0 + t;
                z[i][t] = (col < NR && row < N) ? B[at[i][t] + LDB * col] : 0.0;
            }
        unroll_for<MT>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            apply_step<k, MT>(z, steps + k * MT * TS);
        });
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const int row = 8 * i + n0 + t;
                if (col < NR && row < N) B[at[i][t] + LDB * col] = z[i][t];
            }
    }
    __syncthreads();
}

// A fixed right-hand side without a zero, entries 1 to 2 in size: solved beside the others (the last tile of 8
// columns has room for it in every shape), it shows what an elimination without pivoting did to all unknowns,
// whichever of them the other right-hand sides reach, and also when those are zero.
__device__ __forceinline__ double probe_rhs(int r) {
    const int h = (37 * r + 11) & 63;
    return h < 32 ? 1.0 + h / 32.0 : -1.0 - (h - 32) / 32.0;
}

// Whether x solves A x = probe_rhs as a stable elimination leaves it, over the CTA: for every row the residual is at
// most kProbeError (|A| |x| + |b|) in the largest row sum and entries, and at most kProbeRow of the row's own
// sum_c |a_rc x_c| + |b_r| (where a part of x is large it hides the rows of the others in the first measure; the
// second allows more, since a sound elimination's fill-in exceeds a sparse row's own entries).  Not a number does not
// pass.  red: 4 doubles a warp; every thread returns the answer.
constexpr double kProbeError = 2e-15, kProbeRow = 1e-12;
template <int N, int NT>
__device__ __forceinline__ bool probe_ok(const double *A, const double *x, double *red) {
    double v[3] = {};
    bool row_ok = true;
    for (int r = threadIdx.x; r < N; r += NT) {
        double res = probe_rhs(r), own = fabs(res), as = 0.0;
        for (int c = 0; c < N; c++) {
            const double a = A[r + N * c], xc = x[c];
            res -= a * xc;
            own += fabs(a * xc);
            as += fabs(a);
        }
        row_ok &= fabs(res) <= kProbeRow * own && isfinite(res);
        v[0] = fmax(v[0], fabs(res));
        v[1] = fmax(v[1], as);
        v[2] = fmax(v[2], fabs(x[r]));
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        for (int o = 16; o > 0; o >>= 1) v[k] = fmax(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
        if ((threadIdx.x & 31) == 0) red[4 * (threadIdx.x >> 5) + k] = v[k];
    }
    row_ok = __syncthreads_and(row_ok);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        v[k] = 0.0;
        for (int w = 0; w < NT / 32; w++) v[k] = fmax(v[k], red[4 * w + k]);
    }
    __syncthreads();
    return row_ok && v[0] <= kProbeError * (v[1] * v[2] + 2.0);
}

// Whether X is the inverse of A (N x N, column-major, leading dimension N) as a stable elimination leaves it: for
// every column j and row r, |(A x_j - e_j)_r| <= tol |A_r| |x_j| (row sum, largest entry; not a number is not).
// Every column is looked at, as one of them says nothing about the unknowns that it does not reach.  Tiles of A X
// over the warps, with the norms from the fragments; one barrier, every thread returns the answer.
template <int N, int NT>
__device__ __forceinline__ bool inverse_ok(const double *A, const double *X, double tol) {
    constexpr int TN = (N + 7) / 8, NW = NT / 32;
    const int lane = threadIdx.x & 31, m = lane >> 2, q = lane & 3;
    bool ok = true;
    for (int t = threadIdx.x >> 5; t < TN * TN; t += NW) {
        const int r = 8 * (t % TN) + m, c = 8 * (t / TN) + m;
        double acc[2] = {0.0, 0.0}, as = 0.0, xm = 0.0;
#pragma unroll
        for (int s = 0; s < (N + 3) / 4; s++) {
            const int k = 4 * s + q;
            const double a = r < N && k < N ? A[r + N * k] : 0.0, x = c < N && k < N ? X[k + N * c] : 0.0;
            as += fabs(a);
            xm = fmax(xm, fabs(x));
            dmma(acc, a, x);
        }
        for (int o = 1; o < 4; o <<= 1) {                               // row r's sum, column c's largest entry
            as += __shfl_xor_sync(0xffffffffu, as, o);
            xm = fmax(xm, __shfl_xor_sync(0xffffffffu, xm, o));
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const double xc = __shfl_sync(0xffffffffu, xm, 4 * (2 * q + h));
            const int j = 8 * (t / TN) + 2 * q + h;
            const double res = fabs(acc[h] - (r == j ? 1.0 : 0.0));
            if (r < N && j < N) ok &= isfinite(res) && res <= tol * as * xc;
        }
    }
    return __syncthreads_and(ok);
}

}  // namespace hdgx
