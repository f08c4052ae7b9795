// Per-k kernels of the direct-minimisation and SCF solvers on the FP64 tensor
// cores (mma64.cuh) for the band counts without a register kernel (dm_small.cu
// has 2 <= nb <= 8): one group of ceil(nb / 8) warps per k-point.
//
// What bounds them at nb = 64 is the FP64 rate (8 nb^3 flops a product against
// 16 nb^2 bytes a field); the team kernels they replace read both operands of
// every complex FMA from shared memory.  Measured on a 72 x 72 mesh, nb = 64
// (one product is 10.9 GFLOP, 0.30 ms at the FP64 rate), before -> now, ms:
// density 1.47 -> 0.26 (half a product), trial 9.7 -> 1.02 (an inverse and a
// product), retraction 9.9 -> 0.42, rotation + gradient 2.9 -> 0.91 (two).
// At nb = 9, the most padded size, on 96 x 96, us: trial 74 -> 58, retraction
// 69 -> 30, rotation + gradient 44 -> 42, density 22 -> 20.
#include "common.cuh"
#include "dm.cuh"
#include "dm_mma.cuh"
#include "mma64.cuh"
#include "small_tile.cuh"
#include "team.cuh"

#include <algorithm>
#include <type_traits>

namespace cpphf {

using tile::cp_async16;
using tile::cp_async_commit;
using tile::cp_async_wait_prev;

namespace {

constexpr int kRing = 3;  // 8-row chunks in flight in the rotation

// shared memory of one group
template <int NT>
constexpr size_t rotate_smem() {
    return sizeof(double2) * (MmaGeo<NT>::MAT + kRing * 8 * (size_t)MmaGeo<NT>::LD);
}
template <int NT>
constexpr size_t density_smem() {
    return sizeof(double2) * MmaGeo<NT>::MAT + sizeof(double) * MmaGeo<NT>::NP;  // a multiple of 16
}

constexpr double TINY_REAL = 1.0e-30;  // types.hpp:13
constexpr double LOGIT_CLIP = 1.0e-6;  // types.hpp:14
constexpr double OCC_CLIP = 1.0e-8;    // types.hpp:16

__device__ __forceinline__ double expit(double x) {
    if (x >= 0.0) return 1.0 / (1.0 + exp(-x));
    const double e = exp(x);
    return e / (1.0 + e);
}

// U = (I + tau d / 2)^-1 (I - tau d / 2) = 2 (I + tau d / 2)^-1 - I (d is
// skew-Hermitian; solver_dm.hpp:251-272 in the elimination form) into the
// warps' row tiles and into Us.  Us is the scratch of the elimination first.
template <int NT>
__device__ __forceinline__ void mma_cayley(double2 (&c)[NT][2], const double2* __restrict__ d, double tau, double2* Us,
                                           int nb, int w, int lane) {
    constexpr int LD = MmaGeo<NT>::LD;
    const int row = 8 * w + (lane >> 2), t = lane & 3;
    const double h = 0.5 * tau;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int col = 8 * j + 2 * t + q;
            c[j][q] = cscale(mat_at(d, row, col, nb), h);
            if (row == col) c[j][q].x += 1.0;
        }
    mma_inverse<NT>(c, Us, w, lane);
    group_sync<NT>();  // the last panel is read
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int col = 8 * j + 2 * t + q;
            double2 u = mk(2.0 * c[j][q].x, 2.0 * c[j][q].y);
            if (row == col) u.x -= 1.0;
            c[j][q] = u;
            Us[row * LD + col] = u;
        }
    group_sync<NT>();
}

// diag(U^H Ft U) of one k-point into ds (nb values in shared memory), U in Us;
// part holds NT x NP doubles.
template <int NT>
__device__ __forceinline__ void mma_diag(const double2* __restrict__ Ft, const double2* Us, double* part, double* ds,
                                         int nb, int w, int lane) {
    constexpr int LD = MmaGeo<NT>::LD, NP = MmaGeo<NT>::NP;
    const int r = lane >> 2, t = lane & 3, gt = 32 * w + lane;
    double2 c[NT][2];
    mma_zero<NT>(c);
    mma_rows<NT, NT>(c, RowsFrom(Ft, nb, w, lane), Us, 0, lane);
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int col = 8 * j + 2 * t + q;
            const double2 u = Us[(8 * w + r) * LD + col];
            double v = u.x * c[j][q].x + u.y * c[j][q].y;  // Re(conj(u) (Ft U))
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (r == 0) part[w * NP + col] = v;
        }
    group_sync<NT>();
    for (int i = gt; i < nb; i += MmaGeo<NT>::GT) {
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < NT; ++b) s += part[b * NP + i];
        ds[i] = s;
    }
    group_sync<NT>();
}

template <int NT>
struct CayleySmem {
    static constexpr size_t kU = MmaGeo<NT>::MAT > mma_inverse_elems<NT>() ? MmaGeo<NT>::MAT : mma_inverse_elems<NT>();
    double2 U[kU];
    double part[NT * MmaGeo<NT>::NP], ds[MmaGeo<NT>::NP];
};

// One backtracking trial (solver_dm.hpp:577-589): U(tau) to Uout,
// diag(U^H Ft U) to ew, the free energy by the last block.
template <int NT>
__global__ void __launch_bounds__(MmaGeo<NT>::THREADS, MmaGeo<NT>::BLOCKS)
    k_trial_mma(const double2* __restrict__ dQ, const double2* __restrict__ Ft, const double* __restrict__ p,
                const double* __restrict__ d_p, const double* __restrict__ wt, double* __restrict__ ew,
                double2* __restrict__ Uout, int64_t nk, int nb, double T_r, double shrink, int last_trial,
                double fallback, DmScalars* S) {
    if (S->accepted) return;  // grid-uniform
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ double red[64];
    constexpr int GR = MmaGeo<NT>::GROUPS;
    const int grp = threadIdx.x / MmaGeo<NT>::GT, gt = threadIdx.x % MmaGeo<NT>::GT, w = gt >> 5, lane = gt & 31;
    CayleySmem<NT>& s = reinterpret_cast<CayleySmem<NT>*>(raw)[grp];
    const double tau = S->tau_cur;
    double v[2] = {0.0, 0.0};
    for (int64_t k = (int64_t)blockIdx.x * GR + grp; k < nk; k += (int64_t)gridDim.x * GR) {
        const size_t off = (size_t)k * nb * nb;
        {
            double2 c[NT][2];
            mma_cayley<NT>(c, dQ + off, tau, s.U, nb, w, lane);
            mma_store<NT>(Uout + off, c, nb, w, lane);
        }
        mma_diag<NT>(Ft + off, s.U, s.part, s.ds, nb, w, lane);
        const double wk = wt[k];
        for (int i = gt; i < nb; i += MmaGeo<NT>::GT) {
            const size_t e = (size_t)k * nb + i;
            const double pv = fmin(fmax(p[e] - tau * d_p[e], OCC_CLIP), 1.0 - OCC_CLIP);
            const double di = s.ds[i];
            ew[e] = di;
            v[0] += wk * pv * di;
            v[1] -= wk * (pv * log(pv) + (1.0 - pv) * log1p(-pv));
        }
    }
    double out[2];
    if (reduce_last_block<2>(v, S->part, &S->counter, out, red) && threadIdx.x == 0) {
        const double om = out[0] - fmax(T_r, 1.0e-14) * out[1];
        if (om < S->omega0) {
            S->accepted = 1;
            S->tau_final = tau;
        } else {
            S->tau_cur = tau * shrink;
            if (last_trial) S->tau_final = S->tau0 * fallback;
        }
    }
}

// Retraction Q <- Q U(tau_final) (solver_dm.hpp:590-594): U of the accepted trial
// is read from Uin (eps_work is in ew already); for the fallback step both are
// formed here.  S = null: the plain product Q <- Q Uin.
template <int NT>
__global__ void __launch_bounds__(MmaGeo<NT>::THREADS, MmaGeo<NT>::BLOCKS)
    k_retract_mma(double2* Q, const double2* __restrict__ dQ, const double2* __restrict__ Ft, double* __restrict__ ew,
                  const double2* __restrict__ Uin, int64_t nk, int nb, const DmScalars* S) {
    extern __shared__ __align__(16) unsigned char raw[];
    constexpr int GR = MmaGeo<NT>::GROUPS;
    const int grp = threadIdx.x / MmaGeo<NT>::GT, gt = threadIdx.x % MmaGeo<NT>::GT, w = gt >> 5, lane = gt & 31;
    CayleySmem<NT>& s = reinterpret_cast<CayleySmem<NT>*>(raw)[grp];
    const bool have = !S || S->accepted;
    const double tau = have ? 0.0 : S->tau_final;
    for (int64_t k = (int64_t)blockIdx.x * GR + grp; k < nk; k += (int64_t)gridDim.x * GR) {
        const size_t off = (size_t)k * nb * nb;
        if (have) {
            mma_load_smem<NT>(s.U, Uin + off, nb, gt);
            group_sync<NT>();
        } else {
            {
                double2 c[NT][2];
                mma_cayley<NT>(c, dQ + off, tau, s.U, nb, w, lane);
            }
            mma_diag<NT>(Ft + off, s.U, s.part, s.ds, nb, w, lane);
            for (int i = gt; i < nb; i += MmaGeo<NT>::GT) ew[(size_t)k * nb + i] = s.ds[i];
        }
        double2 c[NT][2];
        mma_zero<NT>(c);
        mma_rows<NT, NT>(c, RowsFrom(Q + off, nb, w, lane), s.U, 0, lane);
        mma_store<NT>(Q + off, c, nb, w, lane);  // a warp reads and writes its own rows only
        group_sync<NT>();
    }
}

// Density P = herm(Q diag(p) Q^H) (solver_dm.hpp:117-128): the tiles (w, w + d mod
// NT), d = 0 .. NT / 2, cover one of each pair of mirrored tiles; the other is
// written as the conjugate transpose, so P is exactly Hermitian.  With mu the
// occupations are p = expit((mu - e) / T) of the energies e, stored to p_out;
// otherwise e holds the occupations.
template <int NT>
__global__ void __launch_bounds__(MmaGeo<NT>::THREADS, MmaGeo<NT>::BLOCKS)
    k_density_mma(const double2* __restrict__ Q, const double* __restrict__ e, const double* __restrict__ mu, double T,
                  double* __restrict__ p_out, double2* __restrict__ P, int64_t nk, int nb) {
    constexpr int LD = MmaGeo<NT>::LD, NP = MmaGeo<NT>::NP, ND = NT / 2 + 1;
    extern __shared__ __align__(16) unsigned char raw[];
    constexpr int GR = MmaGeo<NT>::GROUPS;
    const int grp = threadIdx.x / MmaGeo<NT>::GT, gt = threadIdx.x % MmaGeo<NT>::GT, w = gt >> 5, lane = gt & 31, r = lane >> 2, t = lane & 3;
    double2* Qs = reinterpret_cast<double2*>(raw + density_smem<NT>() * grp);
    double* ps = reinterpret_cast<double*>(Qs + MmaGeo<NT>::MAT);
    const double m = mu ? *mu : 0.0;
    for (int64_t k = (int64_t)blockIdx.x * GR + grp; k < nk; k += (int64_t)gridDim.x * GR) {
        const size_t off = (size_t)k * nb * nb;
        mma_load_smem<NT>(Qs, Q + off, nb, gt);
        for (int i = gt; i < NP; i += MmaGeo<NT>::GT) {
            double pv = 0.0;
            if (i < nb) {
                pv = e[(size_t)k * nb + i];
                if (mu) {
                    pv = expit((m - pv) / T);
                    p_out[(size_t)k * nb + i] = pv;
                }
            }
            ps[i] = pv;
        }
        group_sync<NT>();
        double2 c[ND][2];
        mma_zero<ND>(c);
        const double2* a = Qs + (8 * w + r) * LD + 2 * t;
#pragma unroll 2
        for (int kt = 0; kt < NT; ++kt) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const double2 av = cscale(a[8 * kt + s], ps[8 * kt + 2 * t + s]);
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                    const int jt = w + d < NT ? w + d : w + d - NT;
                    zmma(c[d], av, cconj(Qs[(8 * jt + r) * LD + 8 * kt + 2 * t + s]));
                }
            }
        }
        const int row = 8 * w + r;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            if (NT % 2 == 0 && NT > 1 && d == NT / 2 && w >= NT / 2) continue;  // the mirrored warp has it
            const int jt = w + d < NT ? w + d : w + d - NT;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = 8 * jt + 2 * t + h;
                if (row >= nb || col >= nb || (d == 0 && col < row)) continue;
                double2 x = c[d][h];
                if (row == col) {
                    x.y = 0.0;
                } else {
                    P[off + (size_t)col * nb + row] = cconj(x);
                }
                P[off + (size_t)row * nb + col] = x;
            }
        }
        group_sync<NT>();
    }
}

// Out = Q^H F Q per k (solver_dm.hpp:130-139), Out may alias F; optional eps =
// Re diag(Out).  The rows of F stream through a ring of three 8-row chunks as the
// B operand of S = Q^H F, and S, in registers, is the A operand of S Q, whose
// column tiles are formed in two halves (both products' accumulators at once
// would not fit).  GRAD: also the Riemannian gradient G_ij = (p_j - p_i)
// (Ft_ij + conj Ft_ji) / 2, g_p and the sums behind grad_norm and lam_pc
// (solver_dm.hpp:142-160, 504-519), from the block's rows just written.
template <int NT, bool GRAD>
__global__ void __launch_bounds__(MmaGeo<NT>::THREADS, MmaGeo<NT>::BLOCKS)
    k_rotate_mma(const double2* __restrict__ Q, const double2* F, double2* Out, double* __restrict__ eps,
                 const double* __restrict__ p, const double* __restrict__ wt, double2* __restrict__ G,
                 double* __restrict__ g_p, int64_t nk, int nb, double T_r, double denom_scale, DmScalars* S) {
    constexpr int LD = MmaGeo<NT>::LD, TH = MmaGeo<NT>::GT;
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ double red[64];
    constexpr int GR = MmaGeo<NT>::GROUPS;
    const int grp = threadIdx.x / MmaGeo<NT>::GT, gt = threadIdx.x % MmaGeo<NT>::GT, w = gt >> 5, lane = gt & 31, r = lane >> 2, t = lane & 3;
    double2* Qs = reinterpret_cast<double2*>(raw + rotate_smem<NT>() * grp);
    double2* ring = Qs + MmaGeo<NT>::MAT;
    const double mu = GRAD ? S->mu : 0.0;
    double v[2] = {0.0, 0.0};  // sum w |G|^2, sum eps^2
    for (int i = gt; i < (int)(MmaGeo<NT>::MAT + kRing * 8 * LD); i += TH) Qs[i] = mk(0.0, 0.0);  // the padding
    group_sync<NT>();
    for (int64_t k = (int64_t)blockIdx.x * GR + grp; k < nk; k += (int64_t)gridDim.x * GR) {
        const size_t off = (size_t)k * nb * nb;
        auto chunk = [&](int kt) {
            double2* dst = ring + (kt % kRing) * 8 * LD;
            for (int e = gt; e < 8 * nb; e += TH) {
                const int i = e / nb, j = e - i * nb;
                if (8 * kt + i < nb)
                    cp_async16(dst + i * LD + j, F + off + (size_t)(8 * kt + i) * nb + j);
                else
                    dst[i * LD + j] = mk(0.0, 0.0);
            }
        };
        for (int e = gt; e < nb * nb; e += TH) {
            const int i = e / nb, j = e - i * nb;
            cp_async16(Qs + i * LD + j, Q + off + e);
        }
        chunk(0);
        cp_async_commit();
        if (NT > 1) chunk(1);
        cp_async_commit();
        double2 c[NT][2];
        mma_zero<NT>(c);
#pragma unroll 1
        for (int kt = 0; kt < NT; ++kt) {
            cp_async_wait_prev();
            group_sync<NT>();  // chunk kt has landed for all, chunk kt - 1 is read by all
            if (kt + 2 < NT) chunk(kt + 2);
            cp_async_commit();
            const double2* b = ring + (kt % kRing) * 8 * LD;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const double2 av = cconj(Qs[(8 * kt + 2 * t + s) * LD + 8 * w + r]);
#pragma unroll
                for (int j = 0; j < NT; ++j) zmma(c[j], av, b[(2 * t + s) * LD + 8 * j + r]);
            }
        }
        const int row = 8 * w + r;
        auto half = [&](auto j0c, auto ncc) {
            constexpr int J0 = decltype(j0c)::value, NC = decltype(ncc)::value;
            double2 o[NC][2];
            mma_zero<NC>(o);
            mma_rows_acc<NT, NC>(o, c, Qs, J0, lane);
            if (row < nb) {
#pragma unroll
                for (int j = 0; j < NC; ++j)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int col = 8 * (J0 + j) + 2 * t + h;
                        if (col < nb) {
                            Out[off + (size_t)row * nb + col] = o[j][h];
                            if (eps && row == col) eps[(size_t)k * nb + row] = o[j][h].x;
                        }
                    }
            }
        };
        half(std::integral_constant<int, 0>{}, std::integral_constant<int, (NT + 1) / 2>{});
        if constexpr (NT > 1)
            half(std::integral_constant<int, (NT + 1) / 2>{}, std::integral_constant<int, NT / 2>{});
        group_sync<NT>();  // the block's Out is written, Qs and the ring are read
        if (GRAD) {
            const double wk = wt[k];
            const double* pk = p + (size_t)k * nb;
            for (int e = gt; e < nb * nb; e += TH) {
                const int i = e / nb, j = e - i * nb;
                double2 g = mk(0.0, 0.0);
                if (i != j) {
                    const double dij = 0.5 * (pk[j] - pk[i]);
                    const double2 a = __ldcg(&Out[off + e]), b = __ldcg(&Out[off + (size_t)j * nb + i]);
                    g = mk(dij * (a.x + b.x), dij * (a.y - b.y));
                }
                G[off + e] = g;
                v[0] += wk * (g.x * g.x + g.y * g.y);
            }
            for (int i = gt; i < nb; i += TH) {
                const double ei = __ldcg(&Out[off + (size_t)i * nb + i]).x;
                const double pv = fmin(fmax(pk[i], LOGIT_CLIP), 1.0 - LOGIT_CLIP);
                g_p[(size_t)k * nb + i] = ei + T_r * (log(pv) - log1p(-pv)) - mu;
                v[1] += ei * ei;
            }
        }
    }
    if (GRAD) {
        double out[2];
        if (reduce_last_block<2>(v, S->part, &S->counter, out, red) && threadIdx.x == 0) {
            const int64_t nv = nk * nb;
            S->grad_norm = sqrt(fmax(0.0, out[0]));
            S->lam_pc = fmax(T_r, denom_scale * sqrt(out[1] / (double)(nv > 1 ? nv : 1) + TINY_REAL));
        }
    }
}

// SCF residuals (solver_scf.hpp:64-75, 224-242): sums of w |P_new - D|^2 and of
// w |F D - D F|^2; F and D are Hermitian, so the commutator is X - X^H with X = F D.
template <int NT>
__global__ void __launch_bounds__(MmaGeo<NT>::THREADS, MmaGeo<NT>::BLOCKS)
    k_scf_residuals_mma(const double2* __restrict__ F, const double2* __restrict__ D, const double2* __restrict__ Pn,
                        const double* __restrict__ wt, int64_t nk, int nb, DmScalars* S, double2* __restrict__ comm) {
    constexpr int LD = MmaGeo<NT>::LD;
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ double red[64];
    constexpr int GR = MmaGeo<NT>::GROUPS;
    const int grp = threadIdx.x / MmaGeo<NT>::GT, gt = threadIdx.x % MmaGeo<NT>::GT, w = gt >> 5, lane = gt & 31, r = lane >> 2, t = lane & 3;
    double2* Xs = reinterpret_cast<double2*>(raw) + MmaGeo<NT>::MAT * grp;
    double v[2] = {0.0, 0.0};
    for (int64_t k = (int64_t)blockIdx.x * GR + grp; k < nk; k += (int64_t)gridDim.x * GR) {
        const size_t off = (size_t)k * nb * nb;
        mma_load_smem<NT>(Xs, D + off, nb, gt);
        group_sync<NT>();
        double2 c[NT][2];
        mma_zero<NT>(c);
        mma_rows<NT, NT>(c, RowsFrom(F + off, nb, w, lane), Xs, 0, lane);
        group_sync<NT>();
        const int row = 8 * w + r;
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) Xs[row * LD + 8 * j + 2 * t + h] = c[j][h];
        group_sync<NT>();
        double sd = 0.0, sc = 0.0;
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = 8 * j + 2 * t + h;
                if (row < nb && col < nb) {
                    const size_t e = off + (size_t)row * nb + col;
                    const double2 d = csub(Pn[e], D[e]);
                    const double2 x = csub(c[j][h], cconj(Xs[col * LD + row]));
                    if (comm) comm[e] = x;
                    sd += d.x * d.x + d.y * d.y;
                    sc += x.x * x.x + x.y * x.y;
                }
            }
        const double wk = wt[k];
        v[0] += wk * sd;
        v[1] += wk * sc;
        group_sync<NT>();
    }
    double out[2];
    if (reduce_last_block<2>(v, S->part, &S->counter, out, red) && threadIdx.x == 0) {
        S->grad_norm = out[0];  // density residual^2 * weight_sum
        S->lam_pc = out[1];     // commutator residual^2 * weight_sum
    }
}

// resident CTAs, at most one per k-point and kDmMaxPartials (the reductions' partials)
template <class K>
int resident_ctas(K kern, int threads, size_t smem) {
    raise_smem(kern);
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem);
    (void)cudaGetLastError();
    return std::min(std::max(per, 1) * num_sms(), kDmMaxPartials);
}

#define MMA_LAUNCH(NT, kern, smem, name, ...)                                                            \
    do {                                                                                                 \
        constexpr int GR = MmaGeo<NT>::GROUPS;                                                           \
        static const int ctas = resident_ctas(kern, MmaGeo<NT>::THREADS, GR * (smem));                   \
        kern<<<(unsigned)std::min<int64_t>((nk + GR - 1) / GR, ctas), MmaGeo<NT>::THREADS, GR * (smem),  \
               st>>>(__VA_ARGS__);                                                                       \
        CPPHF_LAUNCH_CHECK(name);                                                                        \
    } while (0)

#define MMA_DISPATCH(nb, X)                                                              \
    switch (((nb) + 7) / 8) {                                                            \
        case 1: X(1); break;                                                             \
        case 2: X(2); break;                                                             \
        case 3: X(3); break;                                                             \
        case 4: X(4); break;                                                             \
        case 5: X(5); break;                                                             \
        case 6: X(6); break;                                                             \
        case 7: X(7); break;                                                             \
        case 8: X(8); break;                                                             \
        case 9: X(9); break;                                                             \
        default: return fail(CPPHF_ERR_UNSUPPORTED, "nb too large for the per-k kernels"); \
    }

}  // namespace

int dm_mma_trial(const double2* dQ, const double2* Ft, const double* p, const double* d_p, const double* w, double* ew,
                 double2* U, int64_t nk, int nb, double T_r, double shrink, int last_trial, double fallback,
                 DmScalars* S, cudaStream_t st) {
#define X(N)                                                                                                     \
    MMA_LAUNCH(N, k_trial_mma<N>, sizeof(CayleySmem<N>), "trial", dQ, Ft, p, d_p, w, ew, U, nk, nb, T_r, shrink, \
               last_trial, fallback, S)
    MMA_DISPATCH(nb, X)
#undef X
    return CPPHF_OK;
}

int dm_mma_retract(double2* Q, const double2* dQ, const double2* Ft, double* ew, const double2* U, int64_t nk, int nb,
                   const DmScalars* S, cudaStream_t st) {
#define X(N) MMA_LAUNCH(N, k_retract_mma<N>, sizeof(CayleySmem<N>), "retract", Q, dQ, Ft, ew, U, nk, nb, S)
    MMA_DISPATCH(nb, X)
#undef X
    return CPPHF_OK;
}

int dm_q_times_u(double2* Q, const double2* U, int64_t nk, int nb, cudaStream_t st) {
    return dm_mma_retract(Q, nullptr, nullptr, nullptr, U, nk, nb, nullptr, st);
}

int dm_mma_density(const double2* Q, const double* e, const double* mu, double T, double* p_out, double2* P, int64_t nk,
                   int nb, cudaStream_t st) {
#define X(N) MMA_LAUNCH(N, k_density_mma<N>, density_smem<N>(), "density", Q, e, mu, T, p_out, P, nk, nb)
    MMA_DISPATCH(nb, X)
#undef X
    return CPPHF_OK;
}

int dm_rotate(const double2* U, const double2* M, double2* Out, double* eps, int64_t nk, int nb, cudaStream_t st) {
#define X(N)                                                                                                  \
    MMA_LAUNCH(N, (k_rotate_mma<N, false>), rotate_smem<N>(), "rotate", U, M, Out, eps, nullptr, nullptr,     \
               nullptr, nullptr, nk, nb, 0.0, 0.0, nullptr)
    MMA_DISPATCH(nb, X)
#undef X
    return CPPHF_OK;
}

int dm_mma_rot_grad(const double2* Q, double2* F, const double* p, const double* w, double* eps, double2* G, double* g_p,
                    int64_t nk, int nb, double T_r, double denom_scale, DmScalars* S, cudaStream_t st) {
#define X(N)                                                                                                       \
    MMA_LAUNCH(N, (k_rotate_mma<N, true>), rotate_smem<N>(), "rotation and gradient", Q, F, F, eps, p, w, G, g_p, \
               nk, nb, T_r, denom_scale, S)
    MMA_DISPATCH(nb, X)
#undef X
    return CPPHF_OK;
}

int scf_mma_residuals(const double2* F, const double2* D, const double2* Pn, const double* w, int64_t nk, int nb,
                      DmScalars* S, double2* comm_out, cudaStream_t st) {
#define X(N)                                                                                                    \
    MMA_LAUNCH(N, k_scf_residuals_mma<N>, sizeof(double2) * MmaGeo<N>::MAT, "scf residuals", F, D, Pn, w, nk, nb, \
               S, comm_out)
    MMA_DISPATCH(nb, X)
#undef X
    return CPPHF_OK;
}

}  // namespace cpphf
