// Batched Hermitian eigendecomposition for small matrices (nb <= 8):
// Householder reduction to real tridiagonal form followed by implicit QL
// iterations, everything in registers (replaces Eigen's SelfAdjointEigenSolver in
// cpp_hf linalg.hpp:39-66, which takes the same tridiagonal + QL route): eight
// lanes per matrix for small batches of nb = 5..8, one thread per matrix
// otherwise, also for the blocks of block-diagonal matrices (k_eigh_thread, below).
//
// Lane r of a group owns column r of A and row r of the accumulated unitary Z.
//  1. Reduction, k = 0 .. nb-3: lane k forms the reflector H = I - beta u u^H
//     that maps A[k+1:, k] to alpha e1 (alpha = -phase(x0) |x|, so the pivot
//     has no cancellation), broadcasts u; every lane j then forms
//     p_j = beta (A u)_j = beta A[:, j]^H u (A is Hermitian), the group sums
//     K = beta/2 u^H p, and with w = p - K u the similarity A <- H A H is the
//     rank-2 update A -= u w^H + w u^H (column j needs w: broadcast).  Z <- Z H
//     is a row-local update.
//  2. A unitary diagonal D (delta_0 = 1, delta_{k+1} = delta_k e_k/|e_k|) makes
//     the tridiagonal real: T' = D^H T D, Z <- Z D.
//  3. Implicit QL with Wilkinson shifts on (d, |e|) (the recurrence of EISPACK's
//     imtql2; Golub & Van Loan, Matrix Computations, sec. 8.3): every lane runs
//     the same scalar recurrence and applies each Givens rotation to its own row
//     of Z.  The matrix is first scaled by a power of two (exact) so that each
//     rotation can use one reciprocal square root.
//  4. Stable ascending sort of the eigenvalues, columns of Z permuted to match.
// Loops over matrix indices are unrolled with compile-time indices so the
// per-lane arrays stay in registers.
#include "common.cuh"
#include "eigh.cuh"

#include <algorithm>
#include <cstdlib>
#include <mutex>

namespace cpphf {

namespace {

constexpr int kHqlThreads = 128;
constexpr int kQlMaxIter = 60;  // QL iterations per eigenvalue before giving up

constexpr int kGroup = 8;  // lanes per matrix of the group form

// Squared norms below this are zero at working precision (the matrices are scaled
// to O(1)); their square roots would have lost their digits to underflow.
constexpr double kTinyNorm2 = 1e-290;
__device__ __forceinline__ double modulus(double2 x) {
    const double m2 = fma(x.x, x.x, x.y * x.y);
    return m2 <= kTinyNorm2 ? 0.0 : sqrt(m2);  // a NaN stays one
}

template <int GS>
__device__ __forceinline__ double group_sum(double v, unsigned mask) {
#pragma unroll
    for (int o = GS / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
}

__device__ __forceinline__ double2 shfl2(double2 v, int src, unsigned mask) {
    return mk(__shfl_sync(mask, v.x, src), __shfl_sync(mask, v.y, src));
}

// four CTAs per SM (<= 128 registers, a few spilled)
template <int NB>
__global__ void __launch_bounds__(kHqlThreads, 4) k_eigh_hql(const double2* __restrict__ M, double* __restrict__ w,
                                                          double2* __restrict__ Vout, int64_t batch, int mode) {
    constexpr int GS = kGroup;
    const int lane = threadIdx.x & 31;
    const int r = lane % GS;
    const int base = lane - r;
    const unsigned mask = (GS == 32 ? 0xffffffffu : (((1u << GS) - 1u) << base));
    const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / GS;
    if (k >= batch) return;  // whole group
    const double2* Mk = M + (size_t)k * NB * NB;

    // column r of herm(M) (mode 0) or herm(i M) (mode 1); lanes r >= NB hold zeros
    double2 a[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        double2 h = mk(0.0, 0.0);
        if (r < NB) {
            double2 x = Mk[i * NB + r], y = Mk[r * NB + i];
            if (mode == 1) {
                x = mk(-x.y, x.x);
                y = mk(-y.y, y.x);
            }
            h = mk(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
            if (i == r) h.y = 0.0;
        }
        a[i] = h;
    }
    // scale by a power of two so the largest entry is O(1): exact, and keeps the
    // QL rotations free of overflow; eigenvalues are scaled back at the end
    double amax = 0.0;
#pragma unroll
    for (int i = 0; i < NB; ++i) amax = fmax(amax, fmax(fabs(a[i].x), fabs(a[i].y)));
#pragma unroll
    for (int o = GS / 2; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(mask, amax, o));
    int ex = 0;
    if (amax > 0.0 && isfinite(amax)) frexp(amax, &ex);
#pragma unroll
    for (int i = 0; i < NB; ++i) a[i] = mk(ldexp(a[i].x, -ex), ldexp(a[i].y, -ex));
    double2 z[NB];  // row r of Z
#pragma unroll
    for (int j = 0; j < NB; ++j) z[j] = mk(j == r ? 1.0 : 0.0, 0.0);

    // ---- 1. Householder reduction ----
#pragma unroll
    for (int kk = 0; kk + 2 < NB; ++kk) {
        // lane kk: reflector of x = A[kk+1:, kk]
        double2 ul[NB];
        double bl = 0.0;
        double2 al = mk(0.0, 0.0);
        if (r == kk) {
            double xn2 = 0.0;
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) xn2 += a[i].x * a[i].x + a[i].y * a[i].y;
            const double2 x0 = a[kk + 1];
            const double ax0 = modulus(x0);
            const double xn = xn2 <= kTinyNorm2 ? 0.0 : sqrt(xn2);
#pragma unroll
            for (int i = 0; i < NB; ++i) ul[i] = mk(0.0, 0.0);
            if (!(xn <= 0.0)) {  // or NaN
                const double iax = ax0 > 0.0 ? 1.0 / ax0 : 0.0;
                const double2 ph = ax0 > 0.0 ? mk(x0.x * iax, x0.y * iax) : mk(1.0, 0.0);
                al = mk(-ph.x * xn, -ph.y * xn);
                ul[kk + 1] = mk(x0.x + ph.x * xn, x0.y + ph.y * xn);
#pragma unroll
                for (int i = kk + 2; i < NB; ++i) ul[i] = a[i];
                bl = 1.0 / (xn * (xn + ax0));
            } else {
                al = x0;
            }
        }
        double2 u[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) u[i] = (i > kk) ? shfl2(ul[i], base + kk, mask) : mk(0.0, 0.0);
        const double beta = __shfl_sync(mask, bl, base + kk);
        const double2 alpha = shfl2(al, base + kk, mask);
        if (beta != 0.0) {  // group-uniform
            // p_r = beta A[:, r]^H u
            double2 pr = mk(0.0, 0.0);
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) cfma(pr, cconj(a[i]), u[i]);
            pr = cscale(pr, beta);
            // K = beta/2 sum_j conj(u_j) p_j (real for Hermitian A)
            double2 ur = u[0];
#pragma unroll
            for (int i = 1; i < NB; ++i)
                if (i == r) ur = u[i];
            if (r >= NB) ur = mk(0.0, 0.0);
            const double Kp = group_sum<GS>(ur.x * pr.x + ur.y * pr.y, mask);
            const double K = 0.5 * beta * Kp;
            const double2 wr = mk(pr.x - K * ur.x, pr.y - K * ur.y);
            double2 wv[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) wv[i] = shfl2(wr, base + i, mask);
            // column r: a -= u conj(w_r) + w conj(u_r)
            const double2 cw = cconj(wr), cu = cconj(ur);
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) {
                a[i] = csub(a[i], cmul(u[i], cw));
                a[i] = csub(a[i], cmul(wv[i], cu));
            }
            // row r of Z: z <- z - beta (z . u) u^H
            double2 t = mk(0.0, 0.0);
#pragma unroll
            for (int j = kk + 1; j < NB; ++j) cfma(t, z[j], u[j]);
            t = cscale(t, beta);
#pragma unroll
            for (int j = kk + 1; j < NB; ++j) z[j] = csub(z[j], cmul(t, cconj(u[j])));
        }
        // exact tridiagonal shape of column / row kk
        if (r == kk) {
            a[kk + 1] = alpha;
#pragma unroll
            for (int i = kk + 2; i < NB; ++i) a[i] = mk(0.0, 0.0);
        } else if (r == kk + 1) {
            a[kk] = cconj(alpha);
        } else if (r > kk + 1) {
            a[kk] = mk(0.0, 0.0);
        }
    }

    // ---- 2. real tridiagonal ----
    double d[NB], e[NB];
    double2 sub[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        double2 di = a[0];
#pragma unroll
        for (int j = 1; j < NB; ++j)
            if (j == i) di = a[j];
        d[i] = __shfl_sync(mask, di.x, base + i);  // A_ii from lane i
        double2 si = mk(0.0, 0.0);
        if (i + 1 < NB) {
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (j == i + 1) si = a[j];
            si = shfl2(si, base + i, mask);  // A_{i+1,i} from lane i
        }
        sub[i] = si;
    }
    double2 delta = mk(1.0, 0.0);
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        z[i] = cmul(z[i], delta);
        if (i + 1 < NB) {
            const double m = modulus(sub[i]);
            e[i] = m;
            if (m > 0.0) {
                const double im = 1.0 / m;
                delta = cmul(delta, mk(sub[i].x * im, sub[i].y * im));
            }
        } else {
            e[i] = 0.0;
        }
    }

    // ---- 3. implicit QL ----
    constexpr double kEps = 2.220446049250313e-16;
    // l unrolled: the sweeps for eigenvalue l address d, e and z at
    // compile-time offsets and issue only the rotations of rows l..NB-2
#pragma unroll
    for (int l = 0; l < NB; ++l) {
        int iter = 0;
        while (true) {
            // first m >= l with a negligible e[m] (m = NB-1 if none)
            int m = NB - 1;
#pragma unroll
            for (int i = NB - 2; i >= 0; --i) {
                if (i >= l) {
                    const double dd = fabs(d[i]) + fabs(d[i + 1]);
                    if (fabs(e[i]) <= kEps * dd) m = i;
                }
            }
            if (m == l || ++iter > kQlMaxIter) break;
            double dl = d[0], dl1 = d[0], el = e[0], dm = d[0];
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                if (j == l) {
                    dl = d[j];
                    el = e[j];
                }
                if (j == l + 1) dl1 = d[j];
                if (j == m) dm = d[j];
            }
            // Wilkinson shift: with t = d[l+1] - d[l], u = 2 e[l] and g0 = t / u,
            // el / (g0 + sign(g0) sqrt(g0^2 + 1)) = el u / (t + sign(t) sqrt(t^2 + u^2)):
            // one division instead of two (the tridiagonal is O(1), so t^2 + u^2
            // can only vanish by underflow; the two-division form covers that case)
            const double t = dl1 - dl, u2 = 2.0 * el;
            const double den = t + copysign(sqrt(fma(t, t, u2 * u2)), t);
            double g;
            if (den != 0.0) {
                g = dm - dl + el * u2 / den;
            } else {
                g = t / u2;
                g = dm - dl + el / (g + copysign(sqrt(fma(g, g, 1.0)), g));
            }
            double rr;
            double s = 1.0, c = 1.0, p = 0.0;
            bool under = false;
#pragma unroll
            for (int i = NB - 2; i >= 0; --i) {
                if (i >= l && i < m && !under) {
                    const double f = s * e[i], b = c * e[i];
                    // Givens pair from one reciprocal square root (the matrix was
                    // scaled to unit size, so f^2 + g^2 cannot overflow)
                    const double q = fma(f, f, g * g);
                    if (q == 0.0) {
                        e[i + 1] = 0.0;
                        d[i + 1] -= p;
                        under = true;
                    } else {
                        const double rinv = rsqrt(q);
                        rr = q * rinv;
                        e[i + 1] = rr;
                        s = f * rinv;
                        c = g * rinv;
                        g = d[i + 1] - p;
                        const double t = (d[i] - g) * s + 2.0 * c * b;
                        p = s * t;
                        d[i + 1] = g + p;
                        g = c * t - b;
                        const double2 zi = z[i], zi1 = z[i + 1];
                        z[i + 1] = mk(s * zi.x + c * zi1.x, s * zi.y + c * zi1.y);
                        z[i] = mk(c * zi.x - s * zi1.x, c * zi.y - s * zi1.y);
                    }
                }
            }
            if (under) {
#pragma unroll
                for (int j = 0; j < NB; ++j)
                    if (j == m) e[j] = 0.0;
                continue;
            }
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                if (j == l) {
                    d[j] -= p;
                    e[j] = g;
                }
                if (j == m) e[j] = 0.0;
            }
        }
    }

    // ---- 4. stable ascending order ----
    int rank[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        int rk = 0;
#pragma unroll
        for (int j = 0; j < NB; ++j)
            if (d[j] < d[i] || (d[j] == d[i] && j < i)) ++rk;
        rank[i] = rk;
    }
    if (r < NB) {
        double2* Vrow = Vout + ((size_t)k * NB + r) * NB;
        double2 out[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            double2 v = z[0];
#pragma unroll
            for (int i = 0; i < NB; ++i)
                if (rank[i] == j) v = z[i];
            out[j] = v;
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) Vrow[j] = out[j];
        if (r == 0) {
            double* wk = w + (size_t)k * NB;
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                double v = d[0];
#pragma unroll
                for (int j = 0; j < NB; ++j)
                    if (rank[j] == i) v = d[j];
                wk[i] = ldexp(v, ex);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Large batches: one thread per matrix, the same reduction and QL.
//
// In the group form every lane repeats the scalar QL recurrence (about forty FP64
// instructions a rotation) to rotate its one row of Z; here a thread runs it once
// and rotates all NB rows of the real eigenvector matrix of the tridiagonal, so
// the FP64 work of a matrix falls to about a third.  The lower triangle of A,
// later Z, fills the registers (two warps per scheduler); the reflectors, scaled
// so that H = I - u u^H, and the phases wait in shared memory.  The columns of Z
// are sorted in registers and transformed two at a time through a padded staging
// tile, so that V is written in whole 32-byte sectors.  The work of a warp is one
// long chain (255 registers, a few spilled at nb = 8), which bounds it up to two
// warps per scheduler; the FP64 pipe does beyond that.  36864 matrices of nb = 8:
// 249 us in groups, 81 us here.
// ---------------------------------------------------------------------------
constexpr int kThreadCta = 64;

template <int NB>
struct ThreadGeo {
    static constexpr int NU = NB * (NB - 1) / 2;               // reflector entries u_k[k+1..NB-1]
    static constexpr int WORDS = 2 * NU + 2 * NB;              // doubles per matrix in shared memory
    static constexpr int STG = 2 * NB + 1;                     // staging stride of a matrix, double2
    static constexpr size_t kSmem = sizeof(double) * WORDS * kThreadCta + sizeof(double2) * STG * kThreadCta;
};

// The diagonal blocks of one size of a batch of ld x ld matrices: problem k is block
// k % count of matrix k / count.
struct BlockClass {
    int ld, count;
    short start[kMaxEighNb];
};

// BLOCKS: the matrices are the diagonal blocks bc, and eigenvalues and vectors go to
// the places of the block (k_block_order then finishes V); a block with a NaN or an
// infinity gives NaN, as eigh_dc does.
template <int NB, bool BLOCKS>
__global__ void __launch_bounds__(kThreadCta, 4)
    k_eigh_thread(const double2* __restrict__ M, double* __restrict__ w, double2* __restrict__ Vout, int64_t batch,
                  int mode, const __grid_constant__ BlockClass bc) {
    using G = ThreadGeo<NB>;
    constexpr bool kNanOut = BLOCKS || NB == 1;
    const int ld = BLOCKS ? bc.ld : NB;
    // element (0, 0) of problem p, and its first eigenvalue
    auto origin = [&](int64_t p) -> size_t {
        if (!BLOCKS) return (size_t)p * NB * NB;
        const int64_t m = p / bc.count;
        return (size_t)m * ld * ld + (size_t)bc.start[p - m * bc.count] * (ld + 1);
    };
    auto first = [&](int64_t p) -> size_t {
        if (!BLOCKS) return (size_t)p * NB;
        const int64_t m = p / bc.count;
        return (size_t)m * ld + bc.start[p - m * bc.count];
    };
    extern __shared__ __align__(16) unsigned char raw[];
    double* sm = reinterpret_cast<double*>(raw) + threadIdx.x;  // word i of the thread at sm[i * kThreadCta]
    const int lane = threadIdx.x & 31, wbase = threadIdx.x - lane;
    double2* stg = reinterpret_cast<double2*>(raw + sizeof(double) * G::WORDS * kThreadCta) + (size_t)wbase * G::STG;
    const int64_t k0 = (int64_t)blockIdx.x * kThreadCta + wbase;  // first matrix of the warp
    if (k0 >= batch) return;
    const int64_t k = min(k0 + lane, batch - 1);  // spare lanes repeat the last matrix
    auto put = [&](int i, double2 v) {
        sm[(2 * i) * kThreadCta] = v.x;
        sm[(2 * i + 1) * kThreadCta] = v.y;
    };
    auto get = [&](int i) { return mk(sm[(2 * i) * kThreadCta], sm[(2 * i + 1) * kThreadCta]); };
    constexpr auto uoff = [](int kk) { return kk * (NB - 1) - kk * (kk - 1) / 2 - (kk + 1); };  // entry of u_kk[i]: + i

    double d[NB], e[NB];
    double nan = 0.0;  // 0, or NaN once an entry is not finite
    int ex = 0;
    {
        // lower triangle of herm(M) or herm(i M), scaled by a power of two
        double2 a[NB][NB];
        const double2* Mk = M + origin(k);
        double amax = 0.0;
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int j = 0; j < NB; ++j) {
                double2 x = Mk[i * ld + j];
                if (mode == 1) x = mk(-x.y, x.x);
                if (j < i) {
                    a[i][j] = x;  // finished when row j's entry (j, i) was read before
                    a[i][j] = mk(0.5 * (x.x + a[j][i].x), 0.5 * (x.y - a[j][i].y));
                } else {
                    a[i][j] = x;
                }
            }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            a[i][i].y = 0.0;
#pragma unroll
            for (int j = 0; j <= i; ++j) {
                amax = fmax(amax, fmax(fabs(a[i][j].x), fabs(a[i][j].y)));
                if (kNanOut) nan += 0.0 * a[i][j].x + 0.0 * a[i][j].y;
            }
        }
        if (amax > 0.0 && isfinite(amax)) frexp(amax, &ex);
        const double sc = ldexp(1.0, -ex);
        // 2^-ex may be subnormal or infinite at the ends of the range: scale in two steps there
        const bool two = !(fabs(sc) >= 2.3e-308 && isfinite(sc));
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int j = 0; j <= i; ++j) {
                if (two)
                    a[i][j] = mk(ldexp(a[i][j].x, -ex), ldexp(a[i][j].y, -ex));
                else
                    a[i][j] = cscale(a[i][j], sc);
            }
        // ---- 1. reduction ----
        double2 sub[NB];
#pragma unroll
        for (int kk = 0; kk + 2 < NB; ++kk) {
            double xn2 = 0.0;
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) xn2 += a[i][kk].x * a[i][kk].x + a[i][kk].y * a[i][kk].y;
            const double2 x0 = a[kk + 1][kk];
            const double ax0 = modulus(x0), xn = sqrt(xn2);
            const bool on = !(xn2 <= kTinyNorm2);  // or NaN
            const double iax = ax0 > 0.0 ? 1.0 / ax0 : 0.0;
            const double2 ph = ax0 > 0.0 ? mk(x0.x * iax, x0.y * iax) : mk(1.0, 0.0);
            // beta = 1 / (xn (xn + ax0)); u is scaled by its square root
            const double rb = on ? rsqrt(xn * (xn + ax0)) : 0.0;
            sub[kk] = on ? mk(-ph.x * xn, -ph.y * xn) : x0;
            double2 u[NB], p[NB];
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) {
                u[i] = i == kk + 1 ? mk((x0.x + ph.x * xn) * rb, (x0.y + ph.y * xn) * rb) : cscale(a[i][kk], rb);
                put(uoff(kk) + i, u[i]);
            }
            double K = 0.0;
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) {
                double2 s = cscale(u[i], a[i][i].x);
#pragma unroll
                for (int j = kk + 1; j < i; ++j) cfma(s, a[i][j], u[j]);
#pragma unroll
                for (int j = i + 1; j < NB; ++j) cfma(s, cconj(a[j][i]), u[j]);
                p[i] = s;
                K += u[i].x * s.x + u[i].y * s.y;
            }
            K *= 0.5;
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) p[i] = mk(p[i].x - K * u[i].x, p[i].y - K * u[i].y);
#pragma unroll
            for (int i = kk + 1; i < NB; ++i)
#pragma unroll
                for (int j = kk + 1; j <= i; ++j) {
                    a[i][j] = csub(a[i][j], cmulc(u[i], p[j]));
                    a[i][j] = csub(a[i][j], cmulc(p[i], u[j]));
                }
        }
        if constexpr (NB >= 2) sub[NB - 2] = a[NB - 1][NB - 2];
        // ---- 2. real tridiagonal ----
        double2 delta = mk(1.0, 0.0);
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            d[i] = a[i][i].x;
            put(G::NU + i, delta);
            e[i] = 0.0;
            if (i + 1 < NB) {
                const double m = modulus(sub[i]);
                e[i] = m;
                if (m > 0.0) {
                    const double im = 1.0 / m;
                    delta = cmul(delta, mk(sub[i].x * im, sub[i].y * im));
                }
            }
        }
    }

    // ---- 3. implicit QL on (d, e) with the real eigenvectors z[row][col] ----
    double z[NB][NB];
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) z[i][j] = i == j ? 1.0 : 0.0;
    constexpr double kEps = 2.220446049250313e-16;
#pragma unroll
    for (int l = 0; l < NB; ++l) {
        for (int iter = 0; iter < kQlMaxIter; ++iter) {
            int m = NB - 1;
#pragma unroll
            for (int i = NB - 2; i >= l; --i)
                if (fabs(e[i]) <= kEps * (fabs(d[i]) + fabs(d[i + 1]))) m = i;
            if (m == l) break;
            double dm = d[NB - 1];
#pragma unroll
            for (int j = l; j < NB; ++j)
                if (j == m) dm = d[j];
            const double el = e[l], t = (l + 1 < NB ? d[l + 1 < NB ? l + 1 : l] : 0.0) - d[l], u2 = 2.0 * el;
            const double den = t + copysign(sqrt(fma(t, t, u2 * u2)), t);
            double g;
            if (den != 0.0) {
                g = dm - d[l] + el * u2 / den;
            } else {
                g = t / u2;
                g = dm - d[l] + el / (g + copysign(sqrt(fma(g, g, 1.0)), g));
            }
            double s = 1.0, c = 1.0, p = 0.0;
            bool under = false;
#pragma unroll
            for (int i = NB - 2; i >= l; --i) {
                if (i < m && !under) {
                    const double f = s * e[i], b = c * e[i], q = fma(f, f, g * g);
                    if (q == 0.0) {
                        e[i + 1] = 0.0;
                        d[i + 1] -= p;
                        under = true;
                    } else {
                        const double rinv = rsqrt(q);
                        e[i + 1] = q * rinv;
                        s = f * rinv;
                        c = g * rinv;
                        g = d[i + 1] - p;
                        const double tt = (d[i] - g) * s + 2.0 * c * b;
                        p = s * tt;
                        d[i + 1] = g + p;
                        g = c * tt - b;
#pragma unroll
                        for (int r = 0; r < NB; ++r) {
                            const double zi = z[r][i], z1 = z[r][i + 1];
                            z[r][i + 1] = s * zi + c * z1;
                            z[r][i] = c * zi - s * z1;
                        }
                    }
                }
            }
            if (!under) {
                d[l] -= p;
                e[l] = g;
            }
#pragma unroll
            for (int j = l; j < NB; ++j)
                if (j == m) e[j] = 0.0;
        }
    }

    // ---- 4. ascending order: odd-even transposition of (d, columns), stable ----
#pragma unroll
    for (int round = 0; round < NB; ++round)
#pragma unroll
        for (int i = round & 1; i + 1 < NB; i += 2) {
            const bool sw = d[i + 1] < d[i];
            const double t = d[i];
            d[i] = sw ? d[i + 1] : t;
            d[i + 1] = sw ? t : d[i + 1];
#pragma unroll
            for (int r = 0; r < NB; ++r) {
                const double x = z[r][i];
                z[r][i] = sw ? z[r][i + 1] : x;
                z[r][i + 1] = sw ? x : z[r][i + 1];
            }
        }
    const int cnt = (int)min((int64_t)32, batch - k0);
    if (lane < cnt) {
#pragma unroll
        for (int i = 0; i < NB; ++i) w[first(k) + i] = ldexp(d[i], ex) + nan;
    }
    // ---- 5. V = H_0 .. H_{NB-3} diag(delta) Z, two columns at a time ----
#pragma unroll
    for (int c0 = 0; c0 < NB; c0 += 2) {
        constexpr int W = 2;
        const int nc = NB - c0 < W ? NB - c0 : W;
        double2 v[W][NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const double2 dl = get(G::NU + i);
#pragma unroll
            for (int c = 0; c < W; ++c) v[c][i] = cscale(dl, z[i][c0 + c < NB ? c0 + c : c0]);
        }
#pragma unroll
        for (int kk = NB - 3; kk >= 0; --kk) {
            double2 t[W];
#pragma unroll
            for (int c = 0; c < W; ++c) t[c] = mk(0.0, 0.0);
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) {
                const double2 u = get(uoff(kk) + i);
#pragma unroll
                for (int c = 0; c < W; ++c) cfma(t[c], cconj(u), v[c][i]);
            }
#pragma unroll
            for (int i = kk + 1; i < NB; ++i) {
                const double2 u = get(uoff(kk) + i);
#pragma unroll
                for (int c = 0; c < W; ++c) v[c][i] = csub(v[c][i], cmul(u, t[c]));
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int c = 0; c < W; ++c) stg[lane * G::STG + 2 * i + c] = kNanOut ? mk(v[c][i].x + nan, v[c][i].y + nan) : v[c][i];
        __syncwarp();
        for (int x = lane; x < cnt * NB * W; x += 32) {
            const int mat = x / (NB * W), r = x - mat * (NB * W), i = r / W, c = r - i * W;
            if (c < nc) Vout[origin(k0 + mat) + (size_t)i * ld + c0 + c] = stg[mat * G::STG + r];
        }
    }
}

template <int NB, bool BLOCKS>
int launch_thread(const double2* M, double* w, double2* V, int64_t batch, int mode, const BlockClass& bc, cudaStream_t st) {
    static std::once_flag once;
    std::call_once(once, [] { raise_smem(k_eigh_thread<NB, BLOCKS>); });
    const unsigned grid = (unsigned)((batch + kThreadCta - 1) / kThreadCta);
    k_eigh_thread<NB, BLOCKS><<<grid, kThreadCta, ThreadGeo<NB>::kSmem, st>>>(M, w, V, batch, mode, bc);
    CPPHF_LAUNCH_CHECK("eigh (thread per matrix)");
    return CPPHF_OK;
}

template <bool BLOCKS>
int thread_per_matrix(int nb, const double2* M, double* w, double2* V, int64_t batch, int mode, const BlockClass& bc,
                      cudaStream_t st) {
    switch (nb) {
        case 1: return launch_thread<1, BLOCKS>(M, w, V, batch, mode, bc, st);
        case 2: return launch_thread<2, BLOCKS>(M, w, V, batch, mode, bc, st);
        case 3: return launch_thread<3, BLOCKS>(M, w, V, batch, mode, bc, st);
        case 4: return launch_thread<4, BLOCKS>(M, w, V, batch, mode, bc, st);
        case 5: return launch_thread<5, BLOCKS>(M, w, V, batch, mode, bc, st);
        case 6: return launch_thread<6, BLOCKS>(M, w, V, batch, mode, bc, st);
        case 7: return launch_thread<7, BLOCKS>(M, w, V, batch, mode, bc, st);
        case 8: return launch_thread<8, BLOCKS>(M, w, V, batch, mode, bc, st);
        default: break;
    }
    return fail(CPPHF_ERR_UNSUPPORTED, "small-matrix eigensolver called with unsupported nb");
}

// A total order of the doubles (NaN included), so that the ranks are a permutation.
__device__ __forceinline__ unsigned long long order_key(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}

// After the blocks of every size: zeros outside the blocks, and with sort the
// eigenvalues ascending over the whole matrix (stable), in place.  A matrix with a
// NaN among its eigenvalues becomes NaN.  Bound by HBM (V read and written once); a CTA
// holds tiles of whole matrices, about kOrderTile entries, in shared memory.
constexpr int kOrderTile = 1024;
constexpr int kOrderThreads = 256;
__host__ __device__ constexpr int order_matrices(int nb) { return nb * nb >= kOrderTile ? 1 : kOrderTile / (nb * nb); }

__global__ void __launch_bounds__(kOrderThreads)
    k_block_order(double* __restrict__ w, double2* __restrict__ V, int64_t batch, int nb, const __grid_constant__ BlockSpec bs) {
    extern __shared__ __align__(16) unsigned char raw[];
    const int nb2 = nb * nb, KT = order_matrices(nb);
    const int64_t k0 = (int64_t)blockIdx.x * KT;
    const int cnt = (int)min((int64_t)KT, batch - k0);
    double2* T = reinterpret_cast<double2*>(raw);
    double* ws = reinterpret_cast<double*>(T + (size_t)KT * nb2);
    int* from = reinterpret_cast<int*>(ws + (size_t)KT * nb);
    int* nan = from + (size_t)KT * nb;
    double2* Vk = V + (size_t)k0 * nb2;
    double* wk = w + (size_t)k0 * nb;
    for (int e = threadIdx.x; e < cnt * nb2; e += kOrderThreads) {
        const int r = e % nb2, i = r / nb, j = r - i * nb;
        T[e] = bs.blk[i] == bs.blk[j] ? Vk[e] : mk(0.0, 0.0);
    }
    for (int e = threadIdx.x; e < cnt; e += kOrderThreads) nan[e] = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < cnt * nb; e += kOrderThreads) {
        ws[e] = wk[e];
        if (isnan(ws[e])) nan[e / nb] = 1;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < cnt * nb; e += kOrderThreads) {
        const int m = e / nb, j = e - m * nb;
        int rank = j;
        if (bs.sort) {
            const unsigned long long kj = order_key(ws[e]);
            rank = 0;
            for (int i = 0; i < nb; ++i) {
                const unsigned long long ki = order_key(ws[m * nb + i]);
                rank += ki < kj || (ki == kj && i < j) ? 1 : 0;
            }
        }
        from[m * nb + rank] = j;
        wk[m * nb + rank] = nan[m] ? NAN : ws[e];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < cnt * nb2; e += kOrderThreads) {
        const int m = e / nb2, r = e - m * nb2, i = r / nb, j = r - i * nb;
        Vk[e] = nan[m] ? mk((double)NAN, (double)NAN) : T[m * nb2 + i * nb + from[m * nb + j]];
    }
}

}  // namespace

bool eigh_small_enabled(int64_t nb) { return nb >= 1 && nb <= 8; }

int eigh_small(const double2* M, double* w, double2* V, int64_t batch, int64_t nb, int mode, cudaStream_t st) {
    // A thread's chain takes 2.6 (nb = 2) to 55 us (nb = 8) however small the batch,
    // and the batch takes little more until every scheduler has two warps; the
    // groups' chains are shorter from nb = 5 on, but their throughput is a third.
    // Measured (thread / group, us): nb = 4 10.6 / 10.7 at 1296 matrices, 13.7 / 28.3
    // at 36864; nb = 6 23.5 / 22.4 at 4608, 23.6 / 25.6 at 6912, 32.7 / 114 at 36864;
    // nb = 8 53.4 / 42.5 at 6912, 52.7 / 53.2 at 9216, 81.4 / 249 at 36864.
    const int64_t least = nb <= 4 ? 0 : nb <= 6 ? 5632 : 9216;
    if (batch >= least) return thread_per_matrix<false>((int)nb, M, w, V, batch, mode, BlockClass(), st);
    const unsigned grid = (unsigned)((batch * kGroup + kHqlThreads - 1) / kHqlThreads);
    switch (nb) {
        case 5: k_eigh_hql<5><<<grid, kHqlThreads, 0, st>>>(M, w, V, batch, mode); break;
        case 6: k_eigh_hql<6><<<grid, kHqlThreads, 0, st>>>(M, w, V, batch, mode); break;
        case 7: k_eigh_hql<7><<<grid, kHqlThreads, 0, st>>>(M, w, V, batch, mode); break;
        case 8: k_eigh_hql<8><<<grid, kHqlThreads, 0, st>>>(M, w, V, batch, mode); break;
        default: return fail(CPPHF_ERR_UNSUPPORTED, "eigh_small: nb out of range");
    }
    CPPHF_LAUNCH_CHECK("eigh (Householder + QL)");
    return CPPHF_OK;
}

// Block by block where every block has a thread kernel.  Measured against eigh_dc on
// whole matrices and the cyclic Jacobi kernel before it (us): 36864 matrices of nb = 8,
// blocks of 2: 28 / 587 / 152, of 4: 51 / 896 / 637; of nb = 4, blocks of 2: 16 / 360 / 76;
// 5184 of nb = 64, blocks of 8: 450 / 3843 / 38900.  A thread's chain for a block of 7
// or 8 is longer than eigh_dc's for up to 16 rows, while that takes one wave (12
// CTAs per SM): 1296 matrices of two blocks of 8 76 / 68, but 5184 80 / 212.
bool eigh_blocks_enabled(int64_t batch, const BlockSpec& bs) {
    if (bs.nblocks <= 1) return false;
    int largest = 0;
    for (int b = 0; b < bs.nblocks; ++b) largest = std::max(largest, bs.start[b + 1] - bs.start[b]);
    if (largest >= 7 && bs.start[bs.nblocks] <= 16 && batch <= 12 * (int64_t)num_sms()) return false;
    return largest <= 8;
}

int eigh_blocks(const double2* M, double* w, double2* V, int64_t batch, int64_t nb, int mode, const BlockSpec& bs,
                cudaStream_t st) {
    for (int size = 1; size <= 8; ++size) {
        BlockClass bc;
        bc.ld = (int)nb;
        bc.count = 0;
        for (int b = 0; b < bs.nblocks; ++b)
            if (bs.start[b + 1] - bs.start[b] == size) bc.start[bc.count++] = bs.start[b];
        if (bc.count) CPPHF_TRY(thread_per_matrix<true>(size, M, w, V, batch * bc.count, mode, bc, st));
    }
    static std::once_flag once;
    std::call_once(once, [] { raise_smem(k_block_order); });
    const size_t KT = (size_t)order_matrices((int)nb);
    const size_t smem = KT * (sizeof(double2) * nb * nb + (sizeof(double) + sizeof(int)) * nb + sizeof(int));
    k_block_order<<<(unsigned)((batch + KT - 1) / KT), kOrderThreads, smem, st>>>(w, V, batch, (int)nb, bs);
    CPPHF_LAUNCH_CHECK("eigh (order of the blocks)");
    return CPPHF_OK;
}

}  // namespace cpphf
