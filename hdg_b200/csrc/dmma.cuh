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

// 1 / x from the hardware's 23-bit approximation (rcp.approx.ftz.f64) and one step of the third-order
// Newton (Householder) iteration y (1 + e + e^2), e = 1 - x y: the relative error goes from 2^-23
// to 2^-69 plus rounding, i.e. within one unit in the last place of the quotient, in three dependent
// operations (the compiled division takes 230 cycles in a dependent chain, this takes about 90).
// A subnormal, zero or non-finite x gives a value that is not finite or not 1 / x: callers check.
__device__ __forceinline__ double fast_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// Inverse of the 8 x 8 matrix held as a C fragment by a warp, in place: Gauss-Jordan over the four
// diagonal 2 x 2 blocks in order (no pivoting).  One 2 x 2 block costs one shuffle round, one
// reciprocal (of its determinant, the products with it formed meanwhile) and two multiply-adds in
// sequence.  Returns false when a determinant is zero or not finite.
__device__ __forceinline__ bool inv8(double (&z)[2]) {
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
        ok &= fabs(det) > 0.0 && isfinite(det);
        const double rd = fast_rcp(det);
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
    __device__ __forceinline__ static int at(int i) { return i; }
};
// Local system of NCU components of NPV nodes (row = node + NPV component): the first two momentum
// components node by node, so that the 2 x 2 pivots of inv8 are a node's, the other components, the
// density last (an interior node has no density pivot before that: the continuity flux does not
// depend on the density).  Without pivoting, largest error of the Jacobian columns over the local
// systems of 2D and 3D Euler and NS states, p = 1 .. 4, against extended precision: 6e-14 (with the
// refined inverses of block_gj); 2e-12 in the order by components with the density last.
template <int NPV, int NCU>
struct PairedOrder {
    __device__ __forceinline__ static int at(int i) {
        return i < 2 * NPV ? NPV * (1 + (i & 1)) + (i >> 1) : (i + NPV < NPV * NCU ? i + NPV : i + NPV - NPV * NCU);
    }
};

// Block Gauss-Jordan elimination of [A | B] (A: N x N, B: N x NR, column-major, leading dimension N)
// without pivoting, in the order Order, B overwritten by the solution, A left as it is; by all NT
// threads.
//
// The transposed system lives in C fragments: warp w holds the columns 8 c .. 8 c + 7 of [A | B] for
// c = w, w + NT / 32, .., as tiles Z(c, i)(m, n) = [A | B](8 i + n, 8 c + m).  A block step k makes
//   Z(c, k) <- Z(c, k) inv(D)^T,   Z(c, i) <- Z(c, i) - Z(c, k) L(i)^T   (i != k)
// with D = A(k, k) and L(i) = A(i, k): the left factor is a tile the warp holds, and a C fragment is
// an A fragment of the columns 2 (l % 4) + s in step s, so no value is exchanged between lanes; the
// right factors are the 8 columns of block k, which their owner has left in shared memory (inv(D)^T
// and -L(i)^T; rows of ten doubles, so that the fragment reads are free of bank conflicts).  While
// the others update, the owner of block k + 1 brings its tile up to date first and inverts the next
// diagonal tile, so one barrier per 8 unknowns remains.  REFINE: the inverse Y of a diagonal tile Q
// gets one Newton step, Y + (I - Y Q) Y.
// What bounds it: the chain of N / 8 inversions (about 1,300 cycles each), with the tensor work of
// other resident elements beside it.  Measured in a loop, cycles per system against an elimination
// of one unknown at a time in registers with a barrier each: N = 40, 49 right-hand sides, three
// CTAs of 192 threads per SM: 31,500 -> 14,200; N = 60, 61, one CTA of 256: 50,200 -> 19,700; N = 50,
// 121, one of 256: 45,700 -> 21,100; N = 24, 37, four of 128: 14,700 -> 6,500 (without REFINE).
// pub: pub_doubles doubles of shared memory, 16-byte aligned, that overlap neither A nor B.
// *bad = 8 k + 1 when block k is singular.
template <int N, int NR, int NT>
struct BlockGJ {
    static constexpr int MT = (N + 7) / 8, RT = (NR + 7) / 8, CT = MT + RT, NW = NT / 32, CPT = (CT + NW - 1) / NW;
    static constexpr int TS = 80, pub_doubles = 2 * MT * TS;
};

template <int N, int NR, int NT, bool REFINE, class Order>
__device__ __forceinline__ void block_gj(const double *__restrict__ A, double *B, double *pub, int *bad) {
    using G = BlockGJ<N, NR, NT>;
    constexpr int MT = G::MT, CT = G::CT, NW = G::NW, CPT = G::CPT, TS = G::TS;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m = lane >> 2, n0 = 2 * (lane & 3);
    double z[CPT][MT][2];
#pragma unroll
    for (int s = 0; s < CPT; s++) {
        const int c = w + s * NW, col = 8 * c + m;
        const double *src = c < MT ? A + N * Order::at(col < N ? col : 0) : B + N * (col - 8 * MT < NR ? col - 8 * MT : 0);
        const bool in = c < MT ? col < N : (c < CT && col - 8 * MT < NR);
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int t = 0; t < 2; t++) {
                const int row = 8 * i + n0 + t;
                z[s][i][t] = (in && row < N) ? src[Order::at(row)] : (c < MT && col == row ? 1.0 : 0.0);
            }
    }
    // the owner of column block k: inverse of its diagonal tile and its other tiles, negated
    auto publish = [&](auto kc) {
        constexpr int k = decltype(kc)::value, s = k / NW;
        double *to = pub + (k & 1) * MT * TS + 10 * m + n0;
        const double *from = pub + (k & 1) * MT * TS + 10 * n0 + m + k * TS;
        double q0 = 0.0, q1 = 0.0;
        if constexpr (REFINE) {                                 // the tile as a right factor
            *reinterpret_cast<double2 *>(to + k * TS) = make_double2(z[s][k][0], z[s][k][1]);
            __syncwarp();
            q0 = from[0];
            q1 = from[10];
        }
        const bool ok = inv8(z[s][k]);
        if (!ok && lane == 0 && *bad == 0) *bad = 8 * k + 1;
        if constexpr (REFINE) {
            double e[2] = {m == n0 ? 1.0 : 0.0, m == n0 + 1 ? 1.0 : 0.0};
            __syncwarp();
            *reinterpret_cast<double2 *>(to + k * TS) = make_double2(z[s][k][0], z[s][k][1]);
            dmma(e, -z[s][k][0], q0);
            dmma(e, -z[s][k][1], q1);
            __syncwarp();
            q0 = from[0];
            q1 = from[10];
            dmma(z[s][k], e[0], q0);
            dmma(z[s][k], e[1], q1);
            __syncwarp();
        }
#pragma unroll
        for (int i = 0; i < MT; i++)
            *reinterpret_cast<double2 *>(to + i * TS) =
                i == k ? make_double2(z[s][i][0], z[s][i][1]) : make_double2(-z[s][i][0], -z[s][i][1]);
    };
    auto step = [&](auto kc) {
        constexpr int k = decltype(kc)::value;
        // right factors: element (row 2 (l % 4) + t, column l / 4) of tile i
        const double *from = pub + (k & 1) * MT * TS + 10 * n0 + m;
        auto update = [&](int s) {
            double p[2] = {0.0, 0.0};
            dmma(p, z[s][k][0], from[k * TS]);
            dmma(p, z[s][k][1], from[k * TS + 10]);
            z[s][k][0] = p[0];
            z[s][k][1] = p[1];
#pragma unroll
            for (int i = 0; i < MT; i++)
                if (i != k) {
                    dmma(z[s][i], p[0], from[i * TS]);
                    dmma(z[s][i], p[1], from[i * TS + 10]);
                }
        };
        constexpr int sn = (k + 1) / NW;                        // the next block's slot in its owner
        const bool next = k + 1 < MT && w == (k + 1) % NW;
        if constexpr (k + 1 < MT) {
            if (next) {
                update(sn);
                publish(std::integral_constant<int, (k + 1 < MT ? k + 1 : 0)>{});
            }
        }
#pragma unroll
        for (int s = 0; s < CPT; s++) {
            const int c = w + s * NW;
            if (c < CT && c > k && !(next && s == sn)) update(s);
        }
        __syncthreads();
    };
    if (w == 0) publish(std::integral_constant<int, 0>{});
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
                    if (row < N) B[Order::at(row) + N * col] = z[s][i][t];
                }
        }
    }
    __syncthreads();
}

}  // namespace hdgx
