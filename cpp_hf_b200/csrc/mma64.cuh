// Complex nb x nb products on the FP64 tensor cores (mma m8n8k4) for the per-k
// kernels of the band counts without a register kernel.
//
// A group of NT warps works on one nb x nb matrix padded to NP = 8 NT (small
// groups share a CTA, each with its own named barrier); warp w of the group owns
// the row tile 8 w .. 8 w + 7 of every result in the accumulator layout: lane
// (r, t) = (lane / 4, lane % 4) holds c[j][h] = element (8 w + r, 8 j + 2 t + h).
// A contraction step (kt, s) of a lane takes the index k = 8 kt + 2 t + s (any
// order of the sum is allowed), so
//   * an accumulator is an A operand as it stands: a(kt, s) = c[kt][s];
//   * row-major operands in shared memory with the odd row stride LD = NP + 1
//     are read without bank conflicts as B, as B^H and as A^H.
// FP64 mma and FP64 FMA have the same rate here (36.9 and 35 TFLOP/s measured),
// but an mma reads each operand element once per eight results: the products
// that read both operands of every FMA from shared memory ran at a tenth of it.
#pragma once

#include "common.cuh"

namespace cpphf {

template <int NT>
struct MmaGeo {
    static constexpr int NP = 8 * NT, LD = NP + 1;
    static constexpr int GT = 32 * NT;  // threads of a group
    // groups of a CTA: the reductions allow 1024 CTAs, too few single-warp ones to fill the SMs
    static constexpr int GROUPS = NT == 1 ? 8 : NT == 2 ? 4 : NT == 3 ? 2 : 1;
    static constexpr int THREADS = GT * GROUPS;
    // CTAs per SM the registers are limited for
    static constexpr int BLOCKS = NT <= 2 ? 3 : NT == 3 ? 4 : NT == 4 ? 5 : NT == 5 ? 4 : NT == 6 ? 3 : NT <= 8 ? 2 : 1;
    static constexpr size_t MAT = (size_t)NP * LD;  // complex elements of one matrix in shared memory
};

// barrier of the calling thread's group
template <int NT>
__device__ __forceinline__ void group_sync() {
    if constexpr (NT == 1) {
        __syncwarp();
    } else if constexpr (MmaGeo<NT>::GROUPS == 1) {
        __syncthreads();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + threadIdx.x / MmaGeo<NT>::GT), "n"(MmaGeo<NT>::GT) : "memory");
    }
}

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}
// c += a b over one complex 8 x 4 by 4 x 8 step
__device__ __forceinline__ void zmma(double2 (&c)[2], double2 a, double2 b) {
    dmma(c[0].x, c[1].x, a.x, b.x);
    dmma(c[0].y, c[1].y, a.x, b.y);
    dmma(c[0].x, c[1].x, -a.y, b.y);
    dmma(c[0].y, c[1].y, a.y, b.x);
}

template <int NT>
__device__ __forceinline__ void mma_zero(double2 (&c)[NT][2]) {
#pragma unroll
    for (int j = 0; j < NT; ++j) c[j][0] = c[j][1] = mk(0.0, 0.0);
}

// element (row, col) of an nb x nb block in global memory, 0 outside
__device__ __forceinline__ double2 mat_at(const double2* X, int row, int col, int nb) {
    return (row < nb && col < nb) ? X[row * nb + col] : mk(0.0, 0.0);
}

// c += A B for row tile w: A from a(kt, s) of the lane (a functor), B row-major in
// shared memory, of which the column tiles J0 .. J0 + NC - 1 are used.
template <int NT, int NC, class FA>
__device__ __forceinline__ void mma_rows(double2 (&c)[NC][2], FA a, const double2* B, int j0, int lane) {
    constexpr int LD = MmaGeo<NT>::LD;
    const int t = lane & 3, n = lane >> 2;
    const double2* b = B + 2 * t * LD + 8 * j0 + n;
    double2 a0 = a(0, 0), a1 = a(0, 1);
#pragma unroll 1
    for (int kt = 0; kt < NT; ++kt, b += 8 * LD) {
        double2 n0 = mk(0.0, 0.0), n1 = mk(0.0, 0.0);
        if (kt + 1 < NT) {
            n0 = a(kt + 1, 0);
            n1 = a(kt + 1, 1);
        }
#pragma unroll
        for (int j = 0; j < NC; ++j) zmma(c[j], a0, b[8 * j]);
#pragma unroll
        for (int j = 0; j < NC; ++j) zmma(c[j], a1, b[LD + 8 * j]);
        a0 = n0;
        a1 = n1;
    }
}

// the same with A in registers (an accumulator of the warp)
template <int NT, int NC>
__device__ __forceinline__ void mma_rows_acc(double2 (&c)[NC][2], const double2 (&a)[NT][2], const double2* B, int j0,
                                             int lane) {
    constexpr int LD = MmaGeo<NT>::LD;
    const double2* b = B + 2 * (lane & 3) * LD + 8 * j0 + (lane >> 2);
#pragma unroll
    for (int kt = 0; kt < NT; ++kt) {
#pragma unroll
        for (int j = 0; j < NC; ++j) zmma(c[j], a[kt][0], b[8 * kt * LD + 8 * j]);
#pragma unroll
        for (int j = 0; j < NC; ++j) zmma(c[j], a[kt][1], b[(8 * kt + 1) * LD + 8 * j]);
    }
}

// functor: rows of an nb x nb matrix in global memory as the A operand of row tile w
struct RowsFrom {
    const double2* X;
    int nb, row, t;
    __device__ RowsFrom(const double2* x, int nb_, int w, int lane) : X(x), nb(nb_), row(8 * w + (lane >> 2)), t(lane & 3) {}
    __device__ __forceinline__ double2 operator()(int kt, int s) const { return mat_at(X, row, 8 * kt + 2 * t + s, nb); }
};

// row tile w of an nb x nb matrix to global memory
template <int NT>
__device__ __forceinline__ void mma_store(double2* X, const double2 (&c)[NT][2], int nb, int w, int lane) {
    const int row = 8 * w + (lane >> 2), t = lane & 3;
    if (row >= nb) return;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (8 * j + 2 * t + h < nb) X[row * nb + 8 * j + 2 * t + h] = c[j][h];
}

// whole nb x nb matrix from global to shared memory, padded with zeros
template <int NT>
__device__ __forceinline__ void mma_load_smem(double2* S, const double2* __restrict__ X, int nb, int tid) {
    using G = MmaGeo<NT>;
    for (int e = tid; e < G::NP * G::NP; e += G::GT) {
        const int i = e / G::NP, j = e - i * G::NP;
        S[i * G::LD + j] = mat_at(X, i, j, nb);
    }
}

// Inverse of an 8 x 8 complex matrix in the accumulator layout of one warp, in
// place, by Gauss-Jordan elimination without pivoting.
__device__ __forceinline__ void inverse8(double2 (&m)[2], int lane) {
    const int r = lane >> 2, t = lane & 3;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const int h = p & 1, src = 4 * p + (p >> 1), own = (lane & 28) + (p >> 1);
        const double2 e = m[h];
        const double2 piv = mk(__shfl_sync(0xffffffffu, e.x, src), __shfl_sync(0xffffffffu, e.y, src));
        const double2 f = mk(__shfl_sync(0xffffffffu, e.x, own), __shfl_sync(0xffffffffu, e.y, own));
        double2 row[2];
#pragma unroll
        for (int c = 0; c < 2; ++c)
            row[c] = mk(__shfl_sync(0xffffffffu, m[c].x, 4 * p + t), __shfl_sync(0xffffffffu, m[c].y, 4 * p + t));
        const double d = 1.0 / (piv.x * piv.x + piv.y * piv.y);
        const double2 inv = mk(piv.x * d, -piv.y * d);
        double2 g = inv;
        if (r != p) {
            g = cmul(f, inv);
            g = mk(-g.x, -g.y);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (2 * t + c == p) {
                m[c] = g;
            } else {
                double2 v = r == p ? mk(0.0, 0.0) : m[c];
                cfma(v, g, row[c]);
                m[c] = v;
            }
        }
    }
}

// Shared scratch of mma_inverse, complex elements: two pivot row panels and two
// 8 x 8 inverses.
template <int NT>
constexpr size_t mma_inverse_elems() {
    return 2 * 8 * (size_t)MmaGeo<NT>::LD + 2 * 8 * 9;
}

// Inverse of an NP x NP matrix with positive definite Hermitian part (no
// pivoting is needed), in place in the warps' row tiles, by blocked Gauss-Jordan
// elimination: per 8-row step the owner warp publishes its raw rows M_p and
// D = M_pp^-1; every other warp i then takes G = -M_ip D and adds G M_p to its
// rows, the owner takes D M_p.  One barrier a step (the panels alternate).
template <int NT>
__device__ __forceinline__ void mma_inverse(double2 (&c)[NT][2], double2* scratch, int w, int lane) {
    constexpr int LD = MmaGeo<NT>::LD;
    const int r = lane >> 2, t = lane & 3;
#pragma unroll
    for (int p = 0; p < NT; ++p) {
        double2* panel = scratch + (p & 1) * 8 * LD;
        double2* D = scratch + 2 * 8 * LD + (p & 1) * 72;
        if (w == p) {
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if (j == p) continue;
                panel[r * LD + 8 * j + 2 * t] = c[j][0];
                panel[r * LD + 8 * j + 2 * t + 1] = c[j][1];
            }
            inverse8(c[p], lane);
            D[r * 9 + 2 * t] = c[p][0];
            D[r * 9 + 2 * t + 1] = c[p][1];
        }
        group_sync<NT>();
        if (w == p) {
#pragma unroll
            for (int j = 0; j < NT; ++j)
                if (j != p) c[j][0] = c[j][1] = mk(0.0, 0.0);
        } else {
            double2 g[2] = {mk(0.0, 0.0), mk(0.0, 0.0)};
#pragma unroll
            for (int s = 0; s < 2; ++s) zmma(g, mk(-c[p][s].x, -c[p][s].y), D[(2 * t + s) * 9 + r]);
            c[p][0] = g[0];
            c[p][1] = g[1];
        }
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int j = 0; j < NT; ++j)
                if (j != p) zmma(c[j], c[p][s], panel[(2 * t + s) * LD + 8 * j + r]);
    }
}

}  // namespace cpphf
