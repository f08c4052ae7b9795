// Chemical-potential solvers as one persistent kernel each (cpp_hf utils.hpp:49-116).
//
// Every block owns a slice of the (nk*nb) eigenvalues.  Per round a block reduces
// its slice (fixed tree), publishes its sums, takes everyone else's and adds all
// of them with the same fixed tree, so the whole grid agrees on (lo, hi, mu) and
// replays the reference's scalar update rule itself.  The results are those of the
// reference's fixed iteration counts (30 bisection steps by default, mu_maxiter
// Newton steps).  Bisection runs its first levels as exact multisection rounds,
// then finds the root of N(mu) = n_e by Newton and replays the remaining levels
// against it (a level whose midpoint lies within the rounding margin of the root is
// counted exactly), which reproduces the bisection's decisions with a few counts
// instead of one per level.  Newton stops early only once its state (mu, lo, hi)
// repeats with period 1 or 2, when the state after the remaining iterations is
// already known.
//
// A round is latency: two exponentials, two block trees and one exchange between
// the blocks.  In the cooperative grid the exchange needs no barrier: each round
// has slots of its own, cleared to a NaN pattern before the launch, a block stores
// its sums into its slot and every block polls all slots until they hold numbers.
// The sums are their own flags, so a round is one store and one L2 round trip
// instead of a counter, a generation word, their fences and a second read.
// Measured against that barrier (bisection / in-loop Newton, us, means of 12
// problems): 1327104 eigenvalues 159 / 98 -> 145 / 91, 294912 82 / 50 -> 68 / 41, 65536
// 143 / 74 -> 106 / 63 (one cluster, its sums in distributed shared memory now), 4608
// 104 / 70 -> 25 / 17 (one block -> one cluster).
#include "common.cuh"
#include "mu.cuh"

#include <mutex>

namespace cpphf {

namespace {

// 512 threads: the shuffles of the two block trees are a third of a round, and
// halve against 1024 (294912 eigenvalues: 71 -> 60 us bisection, 51 -> 35 in-loop)
constexpr int kMuThreads = 512;
constexpr int kMuMaxGrid = 1024;
constexpr int kMuCache = 4;                           // eigenvalues a thread keeps in registers across rounds
// Forms by the number of eigenvalues, each an ordinary launch but the last.
// Measured (bisection / in-loop Newton, us), one block against one cluster: 24.8 /
// 14.5 and 22.8 / 16.5 at 1152 eigenvalues, 53 / 29 and 27 / 16.5 at 4608.  One cluster
// against the cooperative grid, for a solve alone: 43 / 42 and 49 / 21 at 18432, 64 / 54
// and 50 / 47 at 36864, 107 / 60 and 43 / 27 at 65536; for eight in-loop solves on each
// of 16 streams, ms: 1.28 and 1.63, 1.40 and 1.85, 1.44 and 1.48.  Solves that run side
// by side, as a sweep's do, share the SMs in clusters but queue for the whole grid, and
// lose by it up to 2^16; a solve alone would gain from the grid from 2^14 on.
constexpr int64_t kMuOneBlockMax = 1024;              // eigenvalues handled by a single CTA
constexpr int kMuCluster = 8;                         // CTAs of the cluster form (portable cluster size)
constexpr int64_t kMuClusterMax = (int64_t)1 << 16;   // eigenvalues handled by one cluster
constexpr int kBisectLevels = 3;                      // bisection steps per grid barrier
constexpr int kMuNV = (1 << kBisectLevels) - 1;       // midpoints evaluated per barrier
constexpr int kMuSums = (kMuNV + 1) / 2;              // pairs that hold a round's sums
constexpr double kMuWide = 64.0;                      // exact multisection while the bracket exceeds 64 T
constexpr int kMuWarmMaxIter = 8;                     // Newton rounds from a warm start before the cold path
constexpr int kMuSlots = 40;                          // slots of a call (rounds before they are cleared and reused)
// barrier words, then slots of 16 bytes per block (fewer than kMuSlots of them on a grid above 205 blocks)
constexpr size_t kMuWsBytes = 64 + 16 * (size_t)8 * kMuMaxGrid;
constexpr int kMuRootMaxIter = 80;                    // safeguarded Newton rounds (bisection fallback)

__device__ __forceinline__ double expit(double x) {
    if (x >= 0.0) return 1.0 / (1.0 + exp(-x));
    const double e = exp(x);
    return e / (1.0 + e);
}

// a / b from y = 1 / b, q = a y and the residual of q, a correction that leaves the
// rounding of one division (Markstein, IBM J. Res. Dev. 34 (1990) 111).
__device__ __forceinline__ double quotient(double a, double b, double q, double y) { return fma(fma(-q, b, a), y, q); }

// expit(d / T) of a cluster or a grid: the values of the reference's expressions with
// one exponential and one reciprocal.  q = d (1 / T) alone has one rounding more, which
// the exponential multiplies by |q|; a solve that stops on a plateau depends on the
// last bits of N(mu) and has to meet the same occupations in every form.  (With the
// divisions themselves an in-loop solve of 294912 eigenvalues takes 39 us, of 65536 75.)
__device__ __forceinline__ double expit_quotient(double d, double T, double q, double invT) {
    const double x = quotient(d, T, q, invT), e = exp(-fabs(x)), b = 1.0 + e, y = 1.0 / b;
    return x >= 0.0 ? y : quotient(e, b, e * y, y);
}

// Shortcut thresholds on the (approximate) logistic argument x: for x >= 37,
// 1 + exp(-x) rounds to 1 in FP64, so expit(x) is exactly 1; for x <= -50,
// expit(x) < 2e-22 and the term is dropped (far below the rounding of any sum
// of weights it enters).  The approximate argument (difference times the
// reciprocal temperature) is within a few ulp of the exact quotient, far from
// either threshold's margin.
constexpr double kFdOne = 37.0;
constexpr double kFdZero = -50.0;

struct MuArgs {
    const double* eps;
    const double* w;  // per-k weights
    int64_t n;        // nk * nb
    int nb;
    double target;
    const double* mu0;  // device warm start (in-loop Newton; optional for the bisection's root) or null
    double T;
    int maxiter;
    int mode;  // 0 bisection (utils.hpp:49-75), 1 in-loop newton (utils.hpp:79-116)
    double* mu_out;
    double* slots;    // [nslots][grid] pairs: the rounds' published sums
    int nslots;
    unsigned* sync;   // [0] count [1] gen [2] error
    unsigned* err;    // device error word (may be null)
    long long spin_limit;  // grid-barrier poll limit
};

// Element i of a block's slice in band-major order (band = i / nk, k = i % nk):
// the 32 lanes of a warp then hold one band at 32 neighbouring k-points, whose
// eigenvalues mostly fall on the same side of a trial mu, so the shortcut
// branches above stay warp-uniform.  eps is (nk, nb) row-major, w per k.
__device__ __forceinline__ void band_major(const MuArgs& a, unsigned i, unsigned nb, double& wk, double& e) {
    const unsigned nk = (unsigned)(a.n / nb);
    const unsigned band = i / nk, k = i - band * nk;
    wk = a.w[k];
    e = a.eps[(size_t)k * nb + band];
}

// Cluster barrier: every thread of every CTA of the cluster (hardware barrier;
// release / acquire at cluster scope orders the stores to the peers' shared memory).
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();  // the aligned forms want the whole warp
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// v to the place that p has in this block, in the shared memory of block `rank` of the cluster
__device__ __forceinline__ void st_cluster(double2* p, unsigned rank, double2 v) {
    unsigned at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(at), "d"(v.x), "d"(v.y) : "memory");
}

__device__ __forceinline__ double2 ld_slot(const double2* p) {
    double2 v;
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_slot(double2* p, double2 v) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y) : "memory");
}
// the pattern of an empty slot half; no arithmetic result has it
__device__ __forceinline__ bool empty(double x) { return __double_as_longlong(x) == -1LL; }
__device__ __forceinline__ double full(double x) { return empty(x) ? NAN : x; }

// Sums (or maxima) over all eigenvalues, one round at a time, in one block, a
// cooperative grid, or one thread-block cluster (kMuCluster CTAs): every block writes its sums into the shared memory of all
// blocks, double-buffered by round parity, and the hardware cluster barrier stands
// between the writes and the reads, so this form touches no global scratch.
enum class MuForm { kOneBlock, kCluster, kGrid };

template <MuForm FORM>
struct MuSync {
    GridBarrier bar;
    double2* slots;  // [nslots][G]
    int nslots, slot, phase, G;
    double (*red)[32 * kMuNV];  // two trees' scratch, used alternately
    double2* peers;             // cluster form: [2][kMuSums][kMuCluster], the blocks' sums
    int* failed;
    unsigned* err;
    long long limit;
    __device__ void init(const MuArgs& a, double (*scratch)[32 * kMuNV], double2* peer_sums, int* fail_flag) {
        bar.init(a.sync, a.spin_limit, a.err);
        slots = reinterpret_cast<double2*>(a.slots);
        nslots = a.nslots;
        slot = phase = 0;
        G = gridDim.x;
        red = scratch;
        peers = peer_sums;
        failed = fail_flag;
        err = a.err;
        limit = a.spin_limit;
    }
    template <bool MAX>
    static __device__ __forceinline__ double op(double a) {
        return MAX ? warp_max(a) : warp_sum(a);
    }
    // fixed tree over the block; every thread gets the result
    template <int NV, bool MAX>
    __device__ __forceinline__ void tree(double (&v)[NV]) {
        double* s = red[phase & 1];
        ++phase;
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            v[i] = op<MAX>(v[i]);
            if (lane == 0) s[32 * i + wid] = v[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = op<MAX>(lane < kMuThreads / 32 ? s[32 * i + lane] : (MAX ? -INFINITY : 0.0));
    }
    // all blocks' values combined, in every thread; false if a wait gave up
    template <int NV, bool MAX = false>
    __device__ bool reduce(double (&v)[NV]) {
        tree<NV, MAX>(v);
        constexpr int NS = (NV + 1) / 2;
        if constexpr (FORM == MuForm::kOneBlock) {
            return true;
        } else if constexpr (FORM == MuForm::kCluster) {
            // a round's buffer is written again two rounds later, behind the barrier that
            // every reader of this round has passed
            double2* b = peers + (slot & 1) * kMuSums * kMuCluster;
            ++slot;
            if (threadIdx.x < kMuCluster) {
#pragma unroll
                for (int u = 0; u < NS; ++u)
                    st_cluster(&b[u * kMuCluster + blockIdx.x], threadIdx.x, mk(v[2 * u], 2 * u + 1 < NV ? v[2 * u + 1] : 0.0));
            }
            cluster_arrive();
            cluster_wait();
            const int lane = threadIdx.x & 31;  // every warp reads all sums
#pragma unroll
            for (int u = 0; u < NS; ++u) {
                const double2 x = lane < kMuCluster ? b[u * kMuCluster + lane] : mk(MAX ? (double)-INFINITY : 0.0, MAX ? (double)-INFINITY : 0.0);
                v[2 * u] = op<MAX>(x.x);
                if (2 * u + 1 < NV) v[2 * u + 1] = op<MAX>(x.y);
            }
            return true;
        } else {
            if (slot + NS > nslots && !recycle()) return false;
            double2* b = slots + (size_t)slot * G;
            slot += NS;
            if (threadIdx.x == 0) {
#pragma unroll
                for (int u = 0; u < NS; ++u)
                    st_slot(&b[u * G + blockIdx.x], mk(full(v[2 * u]), 2 * u + 1 < NV ? full(v[2 * u + 1]) : 0.0));
            }
#pragma unroll
            for (int i = 0; i < NV; ++i) v[i] = MAX ? -INFINITY : 0.0;
            bool ok = true;
            for (int t = threadIdx.x; t < G && ok; t += kMuThreads) {
#pragma unroll
                for (int u = 0; u < NS; ++u) {
                    double2 x = ld_slot(&b[u * G + t]);
                    for (long long spins = 0; empty(x.x) || empty(x.y); x = ld_slot(&b[u * G + t])) {
                        if (++spins > limit) {
                            ok = false;
                            break;
                        }
                    }
                    v[2 * u] = MAX ? fmax(v[2 * u], x.x) : v[2 * u] + x.x;
                    if (2 * u + 1 < NV) v[2 * u + 1] = MAX ? fmax(v[2 * u + 1], x.y) : v[2 * u + 1] + x.y;
                }
            }
            if (!ok) {
                *failed = 1;
                if (err) atomicOr(err, kWaitErrBarrier);
            }
            tree<NV, MAX>(v);  // its barrier also orders the flag
            return *failed == 0;
        }
    }
    // every slot is used: meet, clear one's own, meet again
    __device__ bool recycle() {
        if (!bar.wait()) return false;
        for (int i = threadIdx.x; i < nslots; i += kMuThreads)
            slots[(size_t)i * G + blockIdx.x] = mk(__longlong_as_double(-1LL), __longlong_as_double(-1LL));
        slot = 0;
        return bar.wait();
    }
};

// kOneBlock is a form of its own for its arithmetic: it keeps the reference's
// expressions as they are written, and a choice between the two at run time costs the
// others 10 to 20 % (in-loop, 294912 eigenvalues: 39 us against 34).
template <MuForm FORM>
__global__ void __launch_bounds__(kMuThreads) k_mu(MuArgs a) {
    constexpr bool CLUSTER = FORM == MuForm::kCluster, one = FORM == MuForm::kOneBlock;
    __shared__ double red[2][32 * kMuNV];
    __shared__ double2 peers[CLUSTER ? 2 * kMuSums * kMuCluster : 1];
    __shared__ int failed;
    if (CLUSTER) cluster_arrive();  // waited for below: no block writes to one that has not started
    if (threadIdx.x == 0) {
        failed = 0;  // ordered by the first tree's barrier
        if (FORM == MuForm::kGrid && blockIdx.x == 0) {
            // barrier words (the launch filled them with the empty pattern): visible before
            // this block's first sums, without which no block comes to use them
            a.sync[0] = a.sync[1] = a.sync[2] = 0u;
            __threadfence();
        }
    }
    MuSync<FORM> net;
    net.init(a, red, peers, &failed);
    const int G = gridDim.x;
    const unsigned nb = (unsigned)a.nb;
    const unsigned n = (unsigned)a.n;
    const unsigned per = (n + G - 1) / G;  // (k, band) elements per block
    const unsigned e0 = blockIdx.x * per;
    const unsigned e1 = min(n, e0 + per);
    // The thread's eigenvalues and weights (band-major), loaded once: with at
    // most kMuCache of them per thread they stay in registers for every round;
    // otherwise every round reloads them.  Same elements, same order either way.
    const bool cached = (per + blockDim.x - 1) / blockDim.x <= (unsigned)kMuCache;  // grid-uniform
    double cw[kMuCache], ce[kMuCache];
#pragma unroll
    for (int u = 0; u < kMuCache; ++u) {
        const unsigned i = e0 + threadIdx.x + u * blockDim.x;
        cw[u] = 0.0;
        ce[u] = 0.0;
        if (cached && i < e1) band_major(a, i, nb, cw[u], ce[u]);
    }
    auto for_each_elem = [&](auto&& f) {
        if (cached) {
#pragma unroll
            for (int u = 0; u < kMuCache; ++u)
                if (e0 + threadIdx.x + u * blockDim.x < e1) f(cw[u], ce[u]);
        } else {
            for (unsigned i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
                double wk, e;
                band_major(a, i, nb, wk, e);
                f(wk, e);
            }
        }
    };
    auto give_up = [&]() {
        if (blockIdx.x == 0 && threadIdx.x == 0) *a.mu_out = NAN;
    };

    // 1. global min / max of eps
    double ends[2] = {-INFINITY, -INFINITY};  // -min, max
    if (cached) {
#pragma unroll
        for (int u = 0; u < kMuCache; ++u)
            if (e0 + threadIdx.x + u * blockDim.x < e1) {
                ends[0] = fmax(ends[0], -ce[u]);
                ends[1] = fmax(ends[1], ce[u]);
            }
    } else {
        for (unsigned i = e0 + threadIdx.x; i < e1; i += blockDim.x) {
            const double e = a.eps[i];
            ends[0] = fmax(ends[0], -e);
            ends[1] = fmax(ends[1], e);
        }
    }
    if (CLUSTER) cluster_wait();
    if (!net.template reduce<2, true>(ends)) return give_up();
    const double emin = -ends[0], emax = ends[1];
    const double Tj = fmax(a.T, 1.0e-12);
    double lo, hi, mu = 0.0;
    if (a.mode == 0) {
        const double span = emax - emin + 10.0 * fmax(Tj, 1.0e-6);
        lo = emin - span;
        hi = emax + span;
    } else {
        lo = emin - 50.0 * Tj;
        hi = emax + 50.0 * Tj;
        mu = fmin(fmax(*a.mu0, lo), hi);
    }
    const double Tfd = Tj + 1.0e-12;  // fermidirac_scalar(x, Tj) = expit(-x / (Tj + 1e-12))
    const double invTfd = 1.0 / Tfd, invTj = 1.0 / Tj;
    if (a.mode == 0) {
        // Bisection (utils.hpp:49-75) in three phases.
        //  1. Exact multisection rounds while the bracket is wide: the counts at
        //     all midpoints of the next kBisectLevels levels of the bisection
        //     tree in one pass, then the tree is walked exactly as the
        //     sequential steps would.
        //  2. The root mu* of N(mu) = target by bracketed Newton from there.
        //  3. The remaining levels replayed against mu*: a midpoint farther than
        //     thr from mu* is decided by comparison (N is increasing, and there
        //     |N(mid) - target| >= 7 eps_N), a nearer one by its exact count.  A
        //     root with thr > T/8 (flat N, e.g. mu in a gap) runs the remaining
        //     levels as exact multisection rounds instead.
        const double epsN = 1.0e-13 * fmax(1.0, fabs(a.target));
        int it = 0;
        double Nlo = NAN, Nhi = NAN;  // counts at the bracket ends when evaluated
        bool ok = true;
        auto msec_round = [&]() {
            const int L = min(kBisectLevels, a.maxiter - it);
            const int nodes = (1 << L) - 1;
            double nlo[kMuNV], nhi[kMuNV], mid[kMuNV];
            nlo[0] = lo;
            nhi[0] = hi;
#pragma unroll
            for (int j = 0; j < kMuNV; ++j) {
                if (j < nodes) {
                    mid[j] = 0.5 * (nlo[j] + nhi[j]);
                    const int l = 2 * j + 1, r = 2 * j + 2;
                    if (l < kMuNV) {
                        nlo[l] = nlo[j];
                        nhi[l] = mid[j];
                    }
                    if (r < kMuNV) {
                        nlo[r] = mid[j];
                        nhi[r] = nhi[j];
                    }
                } else {
                    mid[j] = 0.0;
                }
            }
            double v[kMuNV];
#pragma unroll
            for (int j = 0; j < kMuNV; ++j) v[j] = 0.0;
            for_each_elem([&](double wk, double e) {
#pragma unroll
                for (int j = 0; j < kMuNV; ++j) {
                    if (j < nodes) {
                        // x = (mid - e) / Tfd: the term is exactly wk for x >= 37
                        // and below 2e-22 wk (dropped) for x <= -50
                        const double xa = (mid[j] - e) * invTfd;
                        if (xa >= kFdOne)
                            v[j] += wk;
                        else if (xa > kFdZero)
                            v[j] += wk * (one ? expit((mid[j] - e) / Tfd) : expit_quotient(mid[j] - e, Tfd, xa, invTfd));
                    }
                }
            });
            if (!net.template reduce<kMuNV>(v)) {
                ok = false;
                return;
            }
            int node = 0;
            for (int l = 0; l < L; ++l) {
                double m = mid[0], N = v[0];
#pragma unroll
                for (int j = 1; j < kMuNV; ++j)
                    if (j == node) {
                        m = mid[j];
                        N = v[j];
                    }
                if (N > a.target) {
                    hi = m;
                    Nhi = N;
                    node = 2 * node + 1;
                } else {
                    lo = m;
                    Nlo = N;
                    node = 2 * node + 2;
                }
            }
            it += L;
        };
        // count N and slope Z = dN/dmu at one mu (one grid round)
        auto count_round = [&](double m, double& N, double& Z) {
            double v[2] = {0.0, 0.0};
            for_each_elem([&](double wk, double e) {
                const double xa = (m - e) * invTfd;
                if (xa >= kFdOne) {
                    v[0] += wk;
                } else if (xa > kFdZero) {
                    const double pf = one ? expit((m - e) / Tfd) : expit_quotient(m - e, Tfd, xa, invTfd);
                    v[0] += wk * pf;
                    v[1] += wk * pf * (1.0 - pf) * invTfd;
                }
            });
            if (!net.template reduce<2>(v)) {
                ok = false;
                return;
            }
            N = v[0];
            Z = v[1];
        };
        // safeguarded Newton for the root of N(mu) = target inside [ra, rb]
        struct Root {
            double m, g, slope;
            bool conv;
        };
        auto newton = [&](double m, double ra, double rb, int maxit) {
            Root R{m, INFINITY, 0.0, false};
            for (int r = 0; ok && r < maxit; ++r) {
                double N = 0.0, Z = 0.0;
                count_round(R.m, N, Z);
                if (!ok) break;
                R.g = N - a.target;
                R.slope = Z;
                if (fabs(R.g) <= epsN) {
                    R.conv = true;
                    break;
                }
                if (R.g > 0.0)
                    rb = R.m;
                else
                    ra = R.m;
                double mn = (Z > 0.0) ? R.m - R.g / Z : NAN;
                if (!(mn > ra && mn < rb)) mn = 0.5 * (ra + rb);
                if (mn == R.m) break;
                R.m = mn;
            }
            return R;
        };
        // replay the levels left against the root when its threshold allows
        auto replay = [&](const Root& R) {
            const double thr = (R.conv && R.slope > 0.0) ? 8.0 * (fabs(R.g) + epsN) / R.slope : INFINITY;
            if (!(ok && thr <= 0.125 * Tj)) return false;
            for (; ok && it < a.maxiter; ++it) {
                const double md = 0.5 * (lo + hi);
                bool up;
                if (fabs(md - R.m) > thr) {
                    up = md > R.m;
                } else {
                    double N = 0.0, Z = 0.0;
                    count_round(md, N, Z);
                    up = N > a.target;
                }
                if (up)
                    hi = md;
                else
                    lo = md;
            }
            return true;
        };
        // A warm start (the caller's previous mu, e.g. the last SCF iteration's)
        // inside the initial bracket: Newton from there over the whole bracket and,
        // if it converges, every level replayed from the top.  The levels depend
        // only on the root, so the result is the same as from a cold start.
        bool done = false;
        if (a.mu0 && a.maxiter > 0) {
            const double warm = *a.mu0;
            if (isfinite(warm) && warm > lo && warm < hi) {
                const Root R = newton(warm, lo, hi, kMuWarmMaxIter);
                done = ok && replay(R);
            }
        }
        if (!done && ok) {
            while (ok && it < a.maxiter && (it == 0 || hi - lo > kMuWide * Tj)) msec_round();
            if (ok && it < a.maxiter) {
                // 2. root: secant start inside the bracket, then safeguarded Newton
                double m = 0.5 * (lo + hi);
                if (isfinite(Nlo) && isfinite(Nhi) && Nhi > Nlo) {
                    const double ms = lo + (a.target - Nlo) * (hi - lo) / (Nhi - Nlo);
                    if (ms > lo && ms < hi) m = ms;
                }
                const Root R = newton(m, lo, hi, kMuRootMaxIter);
                // 3. replay, or exact multisection for a flat N
                if (!replay(R))
                    while (ok && it < a.maxiter) msec_round();
            }
        }
        if (!ok) return give_up();
    } else {
        // Newton in a bracket.  The update is a deterministic function of the
        // state (mu, lo, hi); once the state repeats with period 1 or 2 the
        // remaining iterations are known, so the loop stops there with the state
        // the full iteration count would end in.
        double mu1 = NAN, lo1 = NAN, hi1 = NAN;  // state one iteration back
        for (int it = 0; it < a.maxiter; ++it) {
            double v[2] = {0.0, 0.0};
            for_each_elem([&](double wk, double e) {
                // p = expit((mu - e) / Tj) is exactly 1 (and p (1 - p) exactly 0)
                // for an argument >= 37; below -50 both terms are dropped
                const double xa = (mu - e) * invTj;
                if (xa >= kFdOne) {
                    v[0] += wk;
                } else if (xa > kFdZero) {
                    const double p = one ? expit((mu - e) / Tj) : expit_quotient(mu - e, Tj, xa, invTj);
                    const double pq = wk * p * (1.0 - p);
                    v[0] += wk * p;
                    v[1] += one ? pq / Tj : pq;  // the reference's terms, or its sum divided once
                }
            });
            if (!net.template reduce<2>(v)) return give_up();
            const double N = v[0], Z = one ? v[1] : v[1] / Tj;
            const double mu0 = mu, lo0 = lo, hi0 = hi;
            const double g = N - a.target;
            if (g < 0.0) lo = mu;
            if (g > 0.0) hi = mu;
            const double Zs = fmax(Z, 1.0e-18);
            double mn = mu - g / Zs;
            const double mb = 0.5 * (lo + hi);
            if (mn <= lo || mn >= hi) mn = mb;
            mn = fmin(fmax(mn, lo), hi);
            if (!isfinite(mn)) mn = mb;
            mu = mn;
            const int rest = a.maxiter - (it + 1);
            if (mu == mu0 && lo == lo0 && hi == hi0) break;  // fixed point
            if (mu == mu1 && lo == lo1 && hi == hi1) {       // period 2: (s1, s0) repeats
                if (rest & 1) mu = mu0;
                break;
            }
            mu1 = mu0;
            lo1 = lo0;
            hi1 = hi0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.mu_out = (a.mode == 0) ? 0.5 * (lo + hi) : mu;
}

// Largest cooperative grid: the resident blocks of the device, at most kMuMaxGrid.
int max_coop_grid() {
    static int g = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mu<MuForm::kGrid>, kMuThreads, 0);
        if (per < 1) per = 1;
        g = std::min(kMuMaxGrid, per * num_sms());
    });
    return g;
}


// ---------------------------------------------------------------------------
// Allocation-free bisection entry point.  The scratch of its cooperative grid
// (barrier words and slots, the same layout the workspace variant uses) is this
// file-scope array, sized for the largest grid the solver ever launches.  Every
// GPU that loads the library holds it until the process exits; every call of more
// than kMuClusterMax eigenvalues shares it.
// ---------------------------------------------------------------------------
constexpr size_t kMuNoAllocScratchBytes = kMuWsBytes;
static __device__ __align__(256) unsigned char g_mu_noalloc_scratch[kMuNoAllocScratchBytes];

}  // namespace

size_t mu_workspace_bytes(int64_t, int64_t) { return kMuWsBytes; }

int mu_solve(const double* eps, const double* w, int64_t nk, int64_t nb, double target,
             const double* mu0, double T, int maxiter, int mode, double* mu_out, void* ws,
             size_t wsb, cudaStream_t st) {
    if (nk < 1 || nb < 1) return fail(CPPHF_ERR_INVALID, "mu: empty eigenvalue array");
    if (nb > (((int64_t)1 << 31) - 1) / nk) return fail(CPPHF_ERR_INVALID, "mu: more than 2^31-1 eigenvalues");
    if (!eps || !w || !mu_out) return fail(CPPHF_ERR_INVALID, "mu: null pointer");
    if (mode == 1 && !mu0) return fail(CPPHF_ERR_INVALID, "mu: null warm start");
    if (!ws || wsb < mu_workspace_bytes(nk, nb)) return fail(CPPHF_ERR_INVALID, "mu: workspace too small");
    const int64_t n = nk * nb;
    int grid = (int)std::min<int64_t>(max_coop_grid(), (n + kMuThreads * kMuCache / 2 - 1) / (kMuThreads * kMuCache / 2));
    if (grid < 1) grid = 1;
    // small problems: one CTA does it all (its barriers are block-local), launched
    // as an ordinary kernel so that solves on other streams keep running beside it
    if (n <= kMuOneBlockMax) grid = 1;
    MuArgs a;
    a.eps = eps;
    a.w = w;
    a.n = n;
    a.nb = (int)nb;
    a.target = target;
    a.mu0 = mu0;
    a.T = T;
    a.maxiter = maxiter;
    a.mode = mode;
    a.mu_out = mu_out;
    a.sync = reinterpret_cast<unsigned*>(ws);
    a.err = wait_error_word();
    if (!a.err) return CPPHF_ERR_CUDA;
    a.spin_limit = barrier_spin_limit();
    a.slots = reinterpret_cast<double*>(static_cast<unsigned char*>(ws) + 64);
    a.nslots = 0;
    if (grid == 1) {
        k_mu<MuForm::kOneBlock><<<1, kMuThreads, 0, st>>>(a);
        CPPHF_LAUNCH_CHECK("mu (one block)");
        return CPPHF_OK;
    }
    if (n <= kMuClusterMax) {
        // mid-size problems: one cluster of kMuCluster CTAs, hardware cluster
        // barriers between the rounds (no software grid barrier)
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kMuCluster);
        cfg.blockDim = dim3(kMuThreads);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kMuCluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        CPPHF_CUDA(cudaLaunchKernelEx(&cfg, k_mu<MuForm::kCluster>, a));
        return CPPHF_OK;
    }
    a.nslots = (int)std::min<int64_t>(kMuSlots, (int64_t)(kMuWsBytes - 64) / 16 / grid);
    CPPHF_CUDA(cudaMemsetAsync(ws, 0xFF, 64 + 16 * (size_t)a.nslots * grid, st));
    void* args[] = {&a};
    CPPHF_CUDA(cudaLaunchCooperativeKernel((const void*)k_mu<MuForm::kGrid>, dim3(grid), dim3(kMuThreads), args, 0, st));
    return CPPHF_OK;
}

}  // namespace cpphf

extern "C" {

size_t cpphf_mu_workspace_bytes(int64_t nk, int64_t nb) { return cpphf::mu_workspace_bytes(nk, nb); }

int cpphf_find_mu_bisection(const double* eps, const double* weights, int64_t nk, int64_t nb,
                            double n_e, double T, int maxiter, double* mu_out, void* workspace,
                            size_t workspace_bytes, void* stream) {
    if (maxiter <= 0) maxiter = 30;
    return cpphf::mu_solve(eps, weights, nk, nb, n_e, nullptr, T, maxiter, 0, mu_out, workspace,
                           workspace_bytes, static_cast<cudaStream_t>(stream));
}

// The device address of g_mu_noalloc_scratch for the current device.  Host
// code only sees a host-side stand-in for the array under that name, so the
// address is looked up once per device with that device current (first call on
// the device; keep that call outside stream capture) and cached.
static int noalloc_scratch(void** out) {
    static std::mutex mtx;
    static void* ptrs[64] = {nullptr};
    int dev = 0;
    CPPHF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return cpphf::fail(CPPHF_ERR_UNSUPPORTED, "find_mu_bisection_noalloc: device index >= 64");
    std::lock_guard<std::mutex> lock(mtx);
    if (!ptrs[dev]) {
        void* p = nullptr;
        CPPHF_CUDA(cudaGetSymbolAddress(&p, cpphf::g_mu_noalloc_scratch));
        ptrs[dev] = p;
    }
    *out = ptrs[dev];
    return CPPHF_OK;
}

int cpphf_find_mu_bisection_noalloc(const double* eps, const double* weights, int64_t nk, int64_t nb, double n_e,
                                    double T, int maxiter, double* mu_out, void* stream) {
    if (nk < 1 || nb < 1) return cpphf::fail(CPPHF_ERR_INVALID, "mu: empty eigenvalue array");
    if (nb > CPPHF_MU_NOALLOC_MAX_EIGENVALUES / nk)
        return cpphf::fail(CPPHF_ERR_INVALID, "find_mu_bisection_noalloc: nk*nb exceeds the maximum of 2^31-1 eigenvalues");
    void* scratch = nullptr;
    CPPHF_TRY(noalloc_scratch(&scratch));
    if (maxiter <= 0) maxiter = 30;
    return cpphf::mu_solve(eps, weights, nk, nb, n_e, nullptr, T, maxiter, 0, mu_out, scratch,
                           cpphf::kMuNoAllocScratchBytes, static_cast<cudaStream_t>(stream));
}

int cpphf_solve_mu_inloop(const double* eps, const double* w_norm, int64_t nk, int64_t nb,
                          double n_target_norm, const double* mu0, double T, int maxiter,
                          double* mu_out, void* workspace, size_t workspace_bytes, void* stream) {
    return cpphf::mu_solve(eps, w_norm, nk, nb, n_target_norm, mu0, T, maxiter, 1, mu_out, workspace,
                           workspace_bytes, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
