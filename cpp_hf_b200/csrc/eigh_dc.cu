// Batched Hermitian eigendecomposition for any nb <= kMaxEighNb (replaces
// Eigen's SelfAdjointEigenSolver in cpp_hf linalg.hpp:39-120; nb <= 8 and block
// structures of small blocks run eigh_small.cu): Householder
// reduction to a real symmetric tridiagonal, divide and conquer on it, and the
// back-transformation, one CTA per matrix in one launch.
//
// Thread (j, q) = (tid / 4, tid % 4) holds the rows i = 4 ii + q of column j in
// registers, for the matrix during the reduction and for the eigenvectors
// during the back-transformation, so both run on register operands with u and
// p broadcast from shared memory.
//  1. Reduction, k = 0 .. n-3: H = I - beta u u^H maps A[k+1:, k] to alpha e1;
//     with p = beta A u, K = beta/2 u^H p and w = p - K u the similarity is the
//     rank-2 update A -= u w^H + w u^H.  Three block barriers a step.  A unitary
//     diagonal makes the subdiagonal e real and non-negative.
//  2. Divide and conquer (Cuppen 1981; Gu and Eisenstat 1995): T is torn at
//     every off-diagonal, T = diag(d_i - e_{i-1} - e_i) + sum e_i v_i v_i^T, and
//     neighbouring blocks are merged pairwise, all merges of a level at once.
//     A merge diagonalises D + rho z z^T: small z and close D deflate; each
//     other eigenvalue is a root of 1 + rho sum z_i^2 / (d_i - x), found by four
//     lanes as an offset from its nearest pole by the two-pole rational
//     iteration (Li 1993) inside a bisection bracket; z is recomputed from the
//     roots (Loewner's formula), which makes the eigenvectors orthogonal to
//     rounding; the vectors are the product of the old ones with
//     z_i / (d_i - x).  The deflation tolerance, the choice of the root formula in the
//     iteration and its fallback are those of LAPACK's dlaed2 and dlaed4 (LAPACK
//     Working Notes 69 and 89).  No step is a chain longer than one row of the matrix,
//     unlike the n^2 dependent rotations of QL.
//  3. The reflectors are applied to the eigenvectors, stored by ascending
//     eigenvalue (stable) or, with block sizes, block by block.
// What bounds it: the latency of the n reduction steps (three barriers, two square
// roots and a division each) and of the secular iterations, at two CTAs per SM for
// nb = 64.  Measured against the cyclic Jacobi kernel it replaces (Hermitian
// matrices with normal entries): 5184 of nb = 64 5.25 ms (84.7), 5184 of nb = 48
// 2.72 (25.6), 2304 of nb = 32 0.44 (3.28), 9216 of nb = 24 1.05 (7.6), of
// nb = 16 0.44 (1.29), of nb = 10 0.37 (0.48), 1296 of nb = 80 3.20 (39.2).  Walking
// column k in its own four threads instead of taking row k from all columns, and
// loading the operands of one row at a time, took 6.46 ms at nb = 64; unrolling the
// loop over k / 4 (row blocks gone at compile time) 6.6 ms, for the code it makes.
#include "common.cuh"
#include "eigh.cuh"

#include <mutex>

namespace cpphf {

namespace {

constexpr double kEps = 2.220446049250313e-16;
// Squared norms below this are zero at working precision (the matrix is scaled to
// O(1)); their square roots would have lost their digits to underflow.
constexpr double kTinyNorm2 = 1e-290;
__device__ __forceinline__ double modulus(double2 x) {
    const double m2 = fma(x.x, x.x, x.y * x.y);
    return m2 > kTinyNorm2 ? sqrt(m2) : 0.0;
}
constexpr int kSecularMaxIter = 60;  // safeguarded: a bisection of the bracket at worst

template <int NE>
struct DcGeo {
    static constexpr int NR = 4 * NE;                     // rows, rounded up
    static constexpr int NT = 4 * ((NR + 7) / 8 * 8);     // threads: four per column, whole warps
    static constexpr int LD = NR + 1;                     // row stride of Q and S
    // CTAs per SM the registers are limited for (the shared memory allows as many)
    static constexpr int BLOCKS = NE <= 4 ? 12 : NE <= 6 ? 8 : NE <= 8 ? 6 : NE <= 12 ? 3 : NE <= 16 ? 2 : 1;
};

// Shared memory of one matrix.  U holds the reflectors packed by column.
template <int NE>
struct DcSmem {
    static constexpr int NR = DcGeo<NE>::NR, LD = DcGeo<NE>::LD;
    double2 U[NR * (NR - 1) / 2];
    double2 xb[2][NR], wb[NR], sub[NR];
    double Q[NR * LD], S[NR * LD];
    double beta[NR], d[NR], e[NR], z[NR], ds[NR], zs[NR], dk[NR], zk[NR], mu[NR], zh[NR], rc[NR], rs[NR];
    double red[2][DcGeo<NE>::NT / 32], red2[DcGeo<NE>::NT / 32], akk;
    double2 s1;  // (A x)_{k+1}
    int perm[NR], nd[NR], pc[NR], df[NR], org[NR], ra[NR], rb[NR], nrot[NR];
};

__device__ __forceinline__ double quad_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}
__device__ __forceinline__ int quad_sum(int v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}
__device__ __forceinline__ double quad_max(double v) {
    v = fmax(v, __shfl_xor_sync(0xffffffffu, v, 1));
    return fmax(v, __shfl_xor_sync(0xffffffffu, v, 2));
}

// a[i] for a CTA-uniform i: a jump instead of NE selects
template <int NE>
__device__ __forceinline__ double2 pick(const double2 (&a)[NE], int i) {
    double2 v = a[NE - 1];
    switch (i) {
#define X(I) \
    case I: v = a[I < NE ? I : 0]; break;
        X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19)
#undef X
        default: break;
    }
    return v;
}

// Root r of 1 + rho sum_i z_i^2 / (d_i - x), d ascending, as (pole, offset).
// Called by the four lanes of a quad (q = 0..3 each sum every fourth term; the
// xor sums leave the same bits in all four) with `on` false for quads without a
// root, which only take part in the shuffles.
__device__ __forceinline__ void secular_root(const double* d, const double* z, double rho, int r, int k, int q, bool on,
                                             int& org, double& mu) {
    double a = 0.0, b = 0.0;
    org = r;
    mu = 0.0;
    const bool last = r == k - 1;
    {
        // the half of the interval with the root: sign of f at its middle
        const double mid = (on && !last) ? 0.5 * (d[r + 1] - d[r]) : 0.0;
        double s = 0.0;
        if (on)
            for (int i = q; i < k; i += 4) s += last ? z[i] * z[i] : z[i] * z[i] / ((d[i] - d[r]) - mid);
        s = quad_sum(s);
        if (on) {
            if (last) {
                b = rho * s;
                mu = b;
            } else if (1.0 + rho * s >= 0.0) {
                b = mid;
                mu = mid;
            } else {
                org = r + 1;
                a = -mid;
                mu = -mid;
            }
        }
    }
    const double dorg = on ? d[org] : 0.0;
    bool run = on;
    for (int it = 0; it < kSecularMaxIter; ++it) {
        if (!__any_sync(0xffffffffu, run)) break;
        double psi = 0.0, dpsi = 0.0, phi = 0.0, dphi = 0.0;
        if (run) {
            for (int i = q; i < k; i += 4) {
                const double t = 1.0 / ((d[i] - dorg) - mu);
                const double v = rho * z[i] * z[i] * t, dv = v * t;
                if (i <= r) {
                    psi += v;
                    dpsi += dv;
                } else {
                    phi += v;
                    dphi += dv;
                }
            }
        }
        psi = quad_sum(psi);
        dpsi = quad_sum(dpsi);
        phi = quad_sum(phi);
        dphi = quad_sum(dphi);
        if (!run) continue;
        const double w = 1.0 + psi + phi;
        if (!(fabs(w) > kEps * k * (1.0 + fabs(psi) + fabs(phi)))) {
            run = false;
            continue;
        }
        if (w < 0.0)
            a = mu;
        else
            b = mu;
        const double d1 = (d[r] - dorg) - mu;
        double eta;
        if (!last) {
            const double d2 = (d[r + 1] - dorg) - mu;
            const double c = w - d1 * dpsi - d2 * dphi;
            const double A = (d1 + d2) * w - d1 * d2 * (dpsi + dphi), B = d1 * d2 * w;
            const double disc = sqrt(fabs(A * A - 4.0 * B * c));
            eta = c == 0.0 ? B / A : (A <= 0.0 ? (A - disc) / (2.0 * c) : 2.0 * B / (A + disc));
        } else {
            eta = d1 + d1 * d1 * dpsi / (w - d1 * dpsi);
        }
        if (!(w * eta < 0.0)) eta = -w / (dpsi + dphi);
        double next = mu + eta;
        if (!(next > a && next < b)) next = 0.5 * (a + b);
        if (next == mu)
            run = false;
        else
            mu = next;
    }
}

// Input transform: mode 0 -> herm(M), 1 -> herm(i M).
template <int NE>
__global__ void __launch_bounds__(DcGeo<NE>::NT, DcGeo<NE>::BLOCKS)
    k_eigh_dc(const double2* __restrict__ M, double* __restrict__ w, double2* __restrict__ Vout, int n, int mode,
              const BlockSpec bs) {
    constexpr int LD = DcGeo<NE>::LD, NR = DcGeo<NE>::NR, NW = DcGeo<NE>::NT / 32;
    constexpr int RG = NE % 4 == 0 ? 4 : 3;  // row blocks whose operands are loaded together
    extern __shared__ __align__(16) unsigned char smem_raw[];
    DcSmem<NE>& s = *reinterpret_cast<DcSmem<NE>*>(smem_raw);
    const int tid = threadIdx.x, q = tid & 3, j = tid >> 2, warp = tid >> 5, lane = tid & 31;
    const double2* Mk = M + (size_t)blockIdx.x * n * n;
    double* wk = w + (size_t)blockIdx.x * n;
    double2* Vk = Vout + (size_t)blockIdx.x * n * n;

    // ---- load, hermitise, scale by a power of two (exact) to O(1) ----
    double2 a[NE];
    double amax = 0.0;
    bool bad = false;
#pragma unroll
    for (int ii = 0; ii < NE; ++ii) {
        const int i = 4 * ii + q;
        double2 h = mk(0.0, 0.0);
        if (i < n && j < n && !(bs.nblocks > 1 && bs.blk[i] != bs.blk[j])) {
            double2 x = Mk[i * n + j], y = Mk[j * n + i];
            if (mode == 1) {
                x = mk(-x.y, x.x);
                y = mk(-y.y, y.x);
            }
            h = mk(0.5 * (x.x + y.x), i == j ? 0.0 : 0.5 * (x.y - y.y));
            bad = bad || !isfinite(h.x) || !isfinite(h.y);
            amax = fmax(amax, fmax(fabs(h.x), fabs(h.y)));
        }
        a[ii] = h;
    }
    amax = warp_max(amax);
    if (lane == 0) s.red[0][warp] = amax;
    if (__syncthreads_or(bad)) {  // a NaN or infinity: no decomposition
        for (int t = tid; t < n * n; t += blockDim.x) Vk[t] = mk((double)NAN, (double)NAN);
        for (int t = tid; t < n; t += blockDim.x) wk[t] = NAN;
        return;
    }
    for (int t = 0; t < NW; ++t) amax = fmax(amax, s.red[0][t]);
    int ex = 0;
    if (amax > 0.0) frexp(amax, &ex);
    const double sc0 = ldexp(1.0, -(ex / 2)), sc1 = ldexp(1.0, -(ex - ex / 2));
#pragma unroll
    for (int ii = 0; ii < NE; ++ii) {
        // 2^-ex in two factors: it may itself be out of range
        a[ii] = mk(a[ii].x * sc0 * sc1, a[ii].y * sc0 * sc1);
    }
    for (int t = tid; t < NR; t += blockDim.x) s.xb[0][t] = s.xb[1][t] = s.wb[t] = mk(0.0, 0.0);
    __syncthreads();

    // ---- 1. reduction ----
    // A is Hermitian, so column k is the conjugate of row k, one element of it in a
    // thread of every column: x = A[k+1:, k] and its norm need no thread to walk a
    // column.  The product A x runs on the raw x while the first warp forms the
    // reflector u = x + c e_{k+1}; A u = A x + c A[:, k+1] and u^H A u follow from
    // the sums.
    for (int k = 0; k + 2 < n; ++k) {
        const int kb = k >> 2, q2 = k & 3;
        const double2 arow = pick<NE>(a, kb), ay = pick<NE>(a, (k + 1) >> 2);  // rows k and k + 1, where q has them
        double2* x = s.xb[k & 1];
        double2 xj = mk(0.0, 0.0);
        const bool col = j > k && j < n;
        if (warp * 8 + 7 >= k) {
            double v = 0.0;
            if (q == q2) {
                if (col) {
                    xj = cconj(arow);
                    x[j] = xj;
                    v = xj.x * xj.x + xj.y * xj.y;
                } else if (j == k) {
                    s.d[k] = arow.x;
                }
            }
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (lane == q2) s.red[k & 1][warp] = v;
        } else if (lane == 0) {
            s.red[k & 1][warp] = 0.0;
        }
        __syncthreads();
        // the reflector: u = x + c e_{k+1}, beta, and the new subdiagonal
        if (tid == 0) {
            double xn2 = 0.0;
#pragma unroll
            for (int t = 0; t < NW; ++t) xn2 += s.red[k & 1][t];
            const double2 x0 = x[k + 1];
            const double ax0 = modulus(x0), xn = sqrt(xn2);
            const bool some = xn2 > kTinyNorm2;
            const double iax = ax0 > 0.0 ? 1.0 / ax0 : 0.0;
            const double2 ph = ax0 > 0.0 ? mk(x0.x * iax, x0.y * iax) : mk(1.0, 0.0);
            s.beta[k] = some ? 1.0 / (xn * (xn + ax0)) : 0.0;
            s.sub[k] = some ? mk(-ph.x * xn, -ph.y * xn) : x0;
        }
        double2 sj = mk(0.0, 0.0), yj = mk(0.0, 0.0);
        if (warp * 8 + 7 > k) {
            // (A x)_j over the rows below k (x is zero beyond n) and A[k+1, j]
            double2 p0 = mk(0.0, 0.0), p1 = mk(0.0, 0.0);
#pragma unroll
            for (int g = 0; g < NE; g += RG)
                if (g + RG > kb) {
                    double2 xi[RG];
#pragma unroll
                    for (int h = 0; h < RG; ++h) {
                        xi[h] = x[4 * (g + h) + q];
                        if (4 * (g + h) + q <= k) xi[h] = mk(0.0, 0.0);
                    }
#pragma unroll
                    for (int h = 0; h < RG; ++h) cfma((h & 1) ? p1 : p0, cconj(a[g + h]), xi[h]);
                }
            sj = mk(quad_sum(p0.x + p1.x), quad_sum(p0.y + p1.y));
            const int src = (lane & 28) + ((q2 + 1) & 3);
            yj = mk(__shfl_sync(0xffffffffu, ay.x, src), __shfl_sync(0xffffffffu, ay.y, src));
            const int own = (lane & 28) + q2;
            xj = mk(__shfl_sync(0xffffffffu, xj.x, own), __shfl_sync(0xffffffffu, xj.y, own));
            double t = (q == 0 && col) ? xj.x * sj.x + xj.y * sj.y : 0.0;
            t += __shfl_xor_sync(0xffffffffu, t, 4);
            t += __shfl_xor_sync(0xffffffffu, t, 8);
            t += __shfl_xor_sync(0xffffffffu, t, 16);
            if (lane == 0) s.red2[warp] = t;
            if (j == k + 1 && q == 0) {
                s.akk = yj.x;
                s.s1 = sj;
            }
        } else if (lane == 0) {
            s.red2[warp] = 0.0;
        }
        __syncthreads();
        const double beta = s.beta[k];
        double2 uj = mk(0.0, 0.0), wj = mk(0.0, 0.0);
        const double2 c = mk(-s.sub[k].x, -s.sub[k].y);  // phase(x_0) |x|
        if (beta != 0.0 && warp * 8 + 7 > k) {
            double uau = 0.0;
#pragma unroll
            for (int t = 0; t < NW; ++t) uau += s.red2[t];
            const double2 s1 = s.s1;
            uau += 2.0 * (c.x * s1.x + c.y * s1.y) + (c.x * c.x + c.y * c.y) * s.akk;
            const double K = 0.5 * beta * beta * uau;
            if (col) {
                uj = j == k + 1 ? cadd(xj, c) : xj;
                double2 pj = sj;
                cfma(pj, c, cconj(yj));
                wj = mk(beta * pj.x - K * uj.x, beta * pj.y - K * uj.y);
            }
        }
        if (col && q == 0) {
            s.U[k * (n - 1) - k * (k - 1) / 2 + j - k - 1] = uj;
            s.wb[j] = wj;
            if (j == k + 1) x[j] = uj;
        }
        __syncthreads();
        if (beta != 0.0 && col) {
            // A -= u w^H + w u^H; rows up to k take part with garbage: nothing reads them again
            const double2 cw = mk(-wj.x, wj.y), cu = mk(-uj.x, uj.y);
#pragma unroll
            for (int g = 0; g < NE; g += RG)
                if (g + RG > kb) {
                    double2 xi[RG], wi[RG];
#pragma unroll
                    for (int h = 0; h < RG; ++h) {
                        xi[h] = x[4 * (g + h) + q];
                        wi[h] = s.wb[4 * (g + h) + q];
                    }
#pragma unroll
                    for (int h = 0; h < RG; ++h) cfma(a[g + h], xi[h], cw);
#pragma unroll
                    for (int h = 0; h < RG; ++h) cfma(a[g + h], wi[h], cu);
                }
        }
    }
    __syncthreads();
    // the last two diagonal entries and the last subdiagonal
#pragma unroll
    for (int ii = 0; ii < NE; ++ii) {
        const int i = 4 * ii + q;
        if (j < n && j + 2 >= n && i == j) s.d[j] = a[ii].x;
        if (j + 2 == n && i == j + 1) s.sub[j] = a[ii];
    }
    for (int t = tid; t < NR * LD; t += blockDim.x) s.Q[t] = (t % LD == t / LD) ? 1.0 : 0.0;
    __syncthreads();

    // ---- real tridiagonal: e_i = |sub_i|, delta_{i+1} = delta_i sub_i / |sub_i| ----
    double2* delta = s.xb[0];
    if (q == 0 && j < n) {
        double ej = 0.0;
        if (j + 1 < n) ej = modulus(s.sub[j]);
        s.e[j] = ej;
        double2 x = mk(1.0, 0.0);
        if (j > 0) {
            const double2 v = s.sub[j - 1];
            const double m = modulus(v);
            if (m > 0.0) x = mk(v.x / m, v.y / m);
        }
        delta[j] = x;
    }
    __syncthreads();
    for (int st = 1; st < n; st *= 2) {  // inclusive product
        double2 x = mk(1.0, 0.0);
        const bool act = q == 0 && j < n && j >= st;
        if (act) x = cmul(delta[j], delta[j - st]);
        __syncthreads();
        if (act) delta[j] = x;
        __syncthreads();
    }
    if (q == 0 && j < n) {
        const double2 x = delta[j];
        const double m = 1.0 / sqrt(fma(x.x, x.x, x.y * x.y));
        delta[j] = mk(x.x * m, x.y * m);
        s.d[j] = s.d[j] - (j > 0 ? s.e[j - 1] : 0.0) - s.e[j];
    }
    __syncthreads();

    // ---- 2. divide and conquer ----
    for (int half = 1; half < n; half *= 2) {
        const int lo = j / (2 * half) * (2 * half), mid = min(lo + half, n), hi = min(lo + 2 * half, n);
        const bool on = j < n && mid < hi;  // this column's block is merged at this level
        const int len = on ? hi - lo : 0;
        const double rho = on ? 2.0 * s.e[mid - 1] : 0.0;
        const double zj = on ? 0.70710678118654752440 * s.Q[(j < mid ? mid - 1 : mid) * LD + j] : 0.0;
        const double dj = on ? s.d[j] : 0.0;
        if (on && q == 0) s.z[j] = zj;
        __syncthreads();
        int rank = 0;
        double dmax = 0.0, zmax = 0.0;
        for (int i = lo + q; i < lo + len; i += 4) {
            const double di = s.d[i];
            rank += (di < dj || (di == dj && i < j)) ? 1 : 0;
            dmax = fmax(dmax, fabs(di));
            zmax = fmax(zmax, fabs(s.z[i]));
        }
        rank = quad_sum(rank);
        const double tol = 8.0 * kEps * fmax(quad_max(dmax), quad_max(zmax));
        if (on && q == 0) {
            const int at = lo + rank;
            s.ds[at] = dj;
            s.zs[at] = zj;
            s.perm[at] = j;
            s.df[at] = rho * fabs(zj) <= tol;
        }
        if (on && q == 1) s.nrot[j] = 0;
        __syncthreads();
        // from here on j is a position in the sorted order of its block
        bool close = false;
        if (on && q == 0 && !s.df[j]) {
            int pv = j - 1;
            while (pv >= lo && s.df[pv]) --pv;
            if (pv >= lo) {
                const double x = s.zs[pv], c = s.zs[j];
                close = fabs((s.ds[j] - s.ds[pv]) * x * c) <= tol * (x * x + c * c);
            }
        }
        if (__syncthreads_or(close)) {
            // rotate each close pair so that one of its z vanishes (in order: a
            // rotated entry may be close to the next one)
            if (on && q == 0 && j == lo) {
                int pv = -1, nr = 0;
                for (int i = lo; i < hi; ++i) {
                    if (s.df[i]) continue;
                    if (pv >= 0) {
                        double x = s.zs[pv], c = s.zs[i];
                        const double dp = s.ds[pv], di = s.ds[i];
                        if (fabs((di - dp) * x * c) <= tol * (x * x + c * c)) {
                            const double tau = hypot(c, x);
                            c /= tau;
                            x = -x / tau;
                            s.zs[i] = tau;
                            s.zs[pv] = 0.0;
                            s.ds[pv] = dp * c * c + di * x * x;
                            s.ds[i] = dp * x * x + di * c * c;
                            s.df[pv] = 1;
                            s.ra[lo + nr] = s.perm[pv];
                            s.rb[lo + nr] = s.perm[i];
                            s.rc[lo + nr] = c;
                            s.rs[lo + nr] = x;
                            ++nr;
                        }
                    }
                    pv = i;
                }
                s.nrot[lo] = nr;
            }
            __syncthreads();
            if (on && q == 0) {  // row j of the block
                const int nr = s.nrot[lo];
                for (int t = 0; t < nr; ++t) {
                    const int ca = s.ra[lo + t], cb = s.rb[lo + t];
                    const double c = s.rc[lo + t], x = s.rs[lo + t];
                    const double va = s.Q[j * LD + ca], vb = s.Q[j * LD + cb];
                    s.Q[j * LD + ca] = c * va + x * vb;
                    s.Q[j * LD + cb] = c * vb - x * va;
                }
            }
            __syncthreads();
        }
        // positions of the k undeflated entries first, then the deflated ones
        int k = 0, before = 0;
        for (int i = lo + q; i < lo + len; i += 4) {
            const int live = s.df[i] ? 0 : 1;
            k += live;
            before += i < j ? live : 0;
        }
        k = quad_sum(k);
        before = quad_sum(before);
        if (on && q == 0) {
            const bool live = !s.df[j];
            const int at = live ? lo + before : lo + k + (j - lo - before);
            s.nd[at] = j;
            s.pc[at] = s.perm[j];
            if (live) {
                s.dk[at] = s.ds[j];
                s.zk[at] = s.zs[j];
            }
        }
        __syncthreads();
        const int r = j - lo;
        const bool root = on && r < k;
        int org;
        double mu;
        secular_root(s.dk + lo, s.zk + lo, rho, r, k, q, root, org, mu);
        if (root && q == 0) {
            s.org[j] = org;
            s.mu[j] = mu;
        }
        __syncthreads();
        // z from the computed roots: z_i^2 = prod_t (x_t - d_i) / prod_{t != i} (d_t - d_i)
        {
            double pr = 1.0;
            if (root) {
                const double di = s.dk[j];
                for (int t = q; t < k; t += 4) {
                    const double num = (s.dk[lo + s.org[lo + t]] - di) + s.mu[lo + t];
                    pr *= t == r ? num : num / (s.dk[lo + t] - di);
                }
            }
            pr *= __shfl_xor_sync(0xffffffffu, pr, 1);
            pr *= __shfl_xor_sync(0xffffffffu, pr, 2);
            if (root && q == 0) s.zh[j] = copysign(sqrt(fabs(pr)), s.zk[j]);
        }
        __syncthreads();
        double dnew = 0.0;
        {
            double nrm = 0.0;
            if (root) {
                const double dorg = s.dk[lo + org];
                dnew = dorg + mu;
                for (int t = q; t < k; t += 4) {
                    const double v = s.zh[lo + t] / ((s.dk[lo + t] - dorg) - mu);
                    s.S[t * LD + j] = v;
                    nrm += v * v;
                }
            }
            nrm = quad_sum(nrm);
            const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
            if (root)
                for (int t = q; t < k; t += 4) s.S[t * LD + j] *= inv;
        }
        __syncwarp();
        double acc[NE];
#pragma unroll
        for (int ii = 0; ii < NE; ++ii) acc[ii] = 0.0;
        if (root) {
            const bool mixed = s.nrot[lo] > 0;  // a rotation joined columns of both halves
#pragma unroll 4
            for (int t = 0; t < k; ++t) {
                const int c = s.pc[lo + t];
                const double v = s.S[t * LD + j];
                const double* Qc = s.Q + q * LD + c;
                // without rotations column c is zero outside its half
                const int i0 = c < mid || mixed ? lo : mid, i1 = c >= mid || mixed ? hi : mid;
#pragma unroll
                for (int g = 0; g < NE; g += 2)  // rows 4 g .. 4 g + 7 of the four lanes
                    if (4 * g + 8 > i0 && 4 * g < i1) {
                        acc[g] = fma(Qc[4 * g * LD], v, acc[g]);
                        acc[g + 1] = fma(Qc[4 * (g + 1) * LD], v, acc[g + 1]);
                    }
            }
        } else if (on) {
            const int at = s.nd[j], c = s.perm[at];
            dnew = s.ds[at];
#pragma unroll
            for (int ii = 0; ii < NE; ++ii) acc[ii] = s.Q[(4 * ii + q) * LD + c];
        }
        __syncthreads();
        if (on) {
            if (q == 0) s.d[j] = dnew;
#pragma unroll
            for (int ii = 0; ii < NE; ++ii) {
                const int i = 4 * ii + q;
                if (i >= lo && i < hi) s.Q[i * LD + j] = acc[ii];
            }
        }
        __syncthreads();
    }

    // ---- 3. order, back-transformation ----
    const double dj = j < n ? s.d[j] : 0.0;
    int rank = 0;
    if (bs.nblocks > 1 && !bs.sort) {
        // the vectors of a block-diagonal matrix keep to one block each: the block
        // of a vector is that of its largest entry
        if (j < n && q == 0) {
            int im = 0;
            double vm = -1.0;
            for (int i = 0; i < n; ++i)
                if (fabs(s.Q[i * LD + j]) > vm) {
                    vm = fabs(s.Q[i * LD + j]);
                    im = i;
                }
            s.nd[j] = bs.blk[im];
        }
        __syncthreads();
        if (j < n)
            for (int i = q; i < n; i += 4) {
                const double di = s.d[i];
                const int bi = s.nd[i], bj = s.nd[j];
                rank += (bi < bj || (bi == bj && (di < dj || (di == dj && i < j)))) ? 1 : 0;
            }
    } else if (j < n) {
        for (int i = q; i < n; i += 4) {
            const double di = s.d[i];
            rank += (di < dj || (di == dj && i < j)) ? 1 : 0;
        }
    }
    rank = quad_sum(rank);
#pragma unroll
    for (int ii = 0; ii < NE; ++ii) {
        const int i = 4 * ii + q;
        a[ii] = mk(0.0, 0.0);
        if (i < n && j < n) a[ii] = cscale(delta[i], s.Q[i * LD + j]);
    }
    for (int k = n - 3; k >= 0; --k) {
        const double beta = s.beta[k];
        if (beta == 0.0) continue;
        const double2* Uk = s.U + (k * (n - 1) - k * (k - 1) / 2 - (k + 1));
        const int kb = k >> 2;
        double2 t0 = mk(0.0, 0.0), t1 = mk(0.0, 0.0);
#pragma unroll
        for (int g = 0; g < NE; g += RG)
            if (g + RG > kb) {
                double2 u[RG];
#pragma unroll
                for (int h = 0; h < RG; ++h) {
                    const int i = 4 * (g + h) + q;
                    u[h] = (i > k && i < n) ? Uk[i] : mk(0.0, 0.0);
                }
#pragma unroll
                for (int h = 0; h < RG; ++h) cfma((h & 1) ? t1 : t0, cconj(u[h]), a[g + h]);
            }
        const double2 t = mk(-beta * quad_sum(t0.x + t1.x), -beta * quad_sum(t0.y + t1.y));
#pragma unroll
        for (int g = 0; g < NE; g += RG)
            if (g + RG > kb) {
                double2 u[RG];
#pragma unroll
                for (int h = 0; h < RG; ++h) {
                    const int i = 4 * (g + h) + q;
                    u[h] = (i > k && i < n) ? Uk[i] : mk(0.0, 0.0);
                }
#pragma unroll
                for (int h = 0; h < RG; ++h) cfma(a[g + h], u[h], t);
            }
    }
    if (j < n) {
        if (q == 0) wk[rank] = ldexp(dj, ex);
#pragma unroll
        for (int ii = 0; ii < NE; ++ii) {
            const int i = 4 * ii + q;
            if (i < n) Vk[(size_t)i * n + rank] = a[ii];
        }
    }
}

template <int NE>
int launch(const double2* M, double* w, double2* V, int64_t batch, int nb, int mode, const BlockSpec& bs,
           cudaStream_t st) {
    static std::once_flag once;
    std::call_once(once, [] { raise_smem(k_eigh_dc<NE>); });
    k_eigh_dc<NE><<<(unsigned)batch, DcGeo<NE>::NT, sizeof(DcSmem<NE>), st>>>(M, w, V, nb, mode, bs);
    CPPHF_LAUNCH_CHECK("eigh (divide and conquer)");
    return CPPHF_OK;
}

}  // namespace

int eigh_dc(const double2* M, double* w, double2* V, int64_t batch, int64_t nb, int mode, const BlockSpec& bs,
            cudaStream_t st) {
    static_assert(kMaxEighNb <= 80, "largest size class");
    // size classes: a thread holds ceil(nb / 4) rows of its column
    const int n = (int)nb;
    if (n <= 16) return launch<4>(M, w, V, batch, n, mode, bs, st);
    if (n <= 24) return launch<6>(M, w, V, batch, n, mode, bs, st);
    if (n <= 32) return launch<8>(M, w, V, batch, n, mode, bs, st);
    if (n <= 48) return launch<12>(M, w, V, batch, n, mode, bs, st);
    if (n <= 64) return launch<16>(M, w, V, batch, n, mode, bs, st);
    return launch<20>(M, w, V, batch, n, mode, bs, st);
}

}  // namespace cpphf
