// Complex128 exchange passes for line lengths without a four-step codelet:
// mixed-radix Stockham stages with register butterflies (the lengths of odd
// meshes, and of the extended grids of the superlattice exchange).
//
// A tile is one line of n points x CB channels; thread (lane, c) of a CTA owns
// channel c and every L-th butterfly of a stage: R loads, R - 1 twiddles, a
// register DFT of R points, R stores.  The first stage loads from global memory
// and the last one stores to it, so a transform of s stages crosses shared
// memory s - 1 times (two buffers, one barrier a stage); in the columns pass the
// last forward stage, the product with VR and the first inverse stage (the same
// radix) stay in registers.  CTAs are persistent over the tiles, which pays for
// the twiddle table.  A prime factor above 13 is a stage of direct sums over the
// pairs x_i +- x_{P-i}, eight outputs to a thread, on lines that pass through
// shared memory at both ends ("plain" plans, also for single-radix lengths).
//
// The field may be padded: only the first s0 x s1 points of the n0 x n1 mesh
// are stored, the others are zero on input and not wanted on output (the
// superlattice grids are zero-padded to twice their support), so half of the
// rows, and half of the loads and stores of the other passes, fall away.
//
// What bounds it: the FP64 and shared-memory work of the butterflies at two to
// three CTAs per SM.  The stages it replaces formed each output from its R
// inputs separately (R loads and complex FMAs per point and stage) and took few
// channels per CTA.  Measured, us, before -> now: build of 100 x 100, nb = 8
// 105 -> 51; of 180 x 180, nb = 6 293 -> 102; of 97 x 97 (prime), nb = 8
// 280 -> 108; streamed exchange with a 480 x 480 extended grid, 16 plane waves,
// 9160 -> 960 (1505 without the padding rule).
#include "common.cuh"
#include "exchange.cuh"
#include "exchange_pipe.cuh"
#include "exchange_smooth.cuh"
#include "fft_reg.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace cpphf {

namespace {

constexpr int kSmoothThreads = 256;
constexpr int kSmoothMaxStages = 8;
constexpr int kSmoothTile = 2048;  // points x channels of a tile: two buffers of 32 KB

struct SmoothPlan {
    int n, ns;
    int plain;  // lines pass through shared memory at both ends (large primes, single radices)
    int r[kSmoothMaxStages];
};

// register DFT of a prime length above 5: cosine and sine sums of the pairs
// x_i +- x_{P-i}
template <int P, bool INV>
__device__ __forceinline__ void dft_prime(double2 (&x)[P]) {
    constexpr int H = (P - 1) / 2;
    constexpr TwTab<P> T{};
    double2 t[H], s[H];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        t[i] = cadd(x[i + 1], x[P - 1 - i]);
        s[i] = csub(x[i + 1], x[P - 1 - i]);
    }
    const double2 x0 = x[0];
    double2 sum = x0;
#pragma unroll
    for (int i = 0; i < H; ++i) sum = cadd(sum, t[i]);
    x[0] = sum;
#pragma unroll
    for (int m = 1; m <= H; ++m) {
        double2 a = x0, b = mk(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int q = (i + 1) * m % P;
            const double c = T.re[q], d = INV ? -T.im[q] : T.im[q];
            a = mk(fma(c, t[i].x, a.x), fma(c, t[i].y, a.y));
            b = mk(fma(-d, s[i].y, b.x), fma(d, s[i].x, b.y));  // + i d s
        }
        x[m] = cadd(a, b);
        x[P - m] = csub(a, b);
    }
}

template <int R, bool INV>
__device__ __forceinline__ void dft_any(double2 (&x)[R]) {
    if constexpr (R == 7 || R == 11 || R == 13) {
        dft_prime<R, INV>(x);
    } else if constexpr (R == 14) {
        double2 a[7], b[7];
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            a[i] = x[2 * i];
            b[i] = x[2 * i + 1];
        }
        dft_prime<7, INV>(a);
        dft_prime<7, INV>(b);
#pragma unroll
        for (int m = 0; m < 7; ++m) {
            const double2 w = twmul<14, INV>(b[m], m);
            x[m] = cadd(a[m], w);
            x[m + 7] = csub(a[m], w);
        }
    } else {
        dft<R, INV>(x);
    }
}

#define SMOOTH_RADICES(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

template <class F>
__device__ __forceinline__ void with_radix(int r, F&& f) {
    switch (r) {
#define X(R) \
    case R: f(std::integral_constant<int, R>{}); break;
        SMOOTH_RADICES(X)
#undef X
        default: break;
    }
}

// the lane's butterflies of one Stockham stage (see fft.cuh for the index rule)
template <int R, bool INV, class LD, class ST>
__device__ __forceinline__ void stage(int n, int Ns, int lane, int L, const double2* tw, LD&& ld, ST&& st) {
    const int nr = n / R, step = nr / Ns;
    for (int j = lane; j < nr; j += L) {
        const int q = j / Ns, k = j - q * Ns;
        double2 x[R];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = ld(j + i * nr);
        if (Ns > 1) {
            const int a = k * step;
#pragma unroll
            for (int i = 1; i < R; ++i) x[i] = INV ? cmulc(x[i], tw[i * a]) : cmul(x[i], tw[i * a]);
        }
        dft_any<R, INV>(x);
        const int base = q * Ns * R + k;
#pragma unroll
        for (int m = 0; m < R; ++m) st(base + m * Ns, x[m]);
    }
}

// One Stockham stage of an odd prime radix P between two tile buffers: X_m and
// X_{P-m} are A +- B with A = x_0 + sum cos (x_i + x_{P-i}), B = i sum sin
// (x_i - x_{P-i}); a thread forms four such pairs of outputs, so a point is read
// once for eight of them.
template <bool INV>
__device__ __forceinline__ void stage_prime(int P, int n, int Ns, int lane, int L, int CB, int c, const double2* tw,
                                            const double2* src, double2* dst) {
    const int nr = n / P, step = nr / Ns, H = (P - 1) / 2, nblk = (H + 3) / 4;
    for (int it = lane; it < nr * nblk; it += L) {
        const int j = it / nblk, m0 = 1 + 4 * (it - j * nblk), q = j / Ns, k = j - q * Ns;
        double2 sum = src[j * CB + c], A[4], B[4];
        int idx[4], m[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            A[b] = sum;
            B[b] = mk(0.0, 0.0);
            m[b] = min(m0 + b, H);
            idx[b] = 0;
        }
        for (int i = 1; i <= H; ++i) {
            double2 u = src[(j + i * nr) * CB + c], v = src[(j + (P - i) * nr) * CB + c];
            if (Ns > 1) {
                const double2 wu = tw[i * k * step], wv = tw[(P - i) * k * step];
                u = INV ? cmulc(u, wu) : cmul(u, wu);
                v = INV ? cmulc(v, wv) : cmul(v, wv);
            }
            const double2 t = cadd(u, v), s = csub(u, v);
            sum = cadd(sum, t);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                idx[b] += m[b];
                if (idx[b] >= P) idx[b] -= P;
                const double2 w = tw[idx[b] * nr];
                const double d = INV ? -w.y : w.y;
                A[b] = mk(fma(w.x, t.x, A[b].x), fma(w.x, t.y, A[b].y));
                B[b] = mk(fma(-d, s.y, B[b].x), fma(d, s.x, B[b].y));
            }
        }
        const int base = q * Ns * P + k;
        if (m0 == 1) dst[base * CB + c] = sum;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            if (m0 + b > H) continue;
            dst[(base + m[b] * Ns) * CB + c] = cadd(A[b], B[b]);
            dst[(base + (P - m[b]) * Ns) * CB + c] = csub(A[b], B[b]);
        }
    }
}

// shared memory: tw[n] | a[n][CB] | b[n][CB]
struct Tile {
    double2 *tw, *a, *b;
    int c, lane, L;
    __device__ Tile(unsigned char* raw, int n, int CB) {
        tw = reinterpret_cast<double2*>(raw);
        a = tw + n;
        b = a + (size_t)n * CB;
        c = threadIdx.x % CB;
        lane = threadIdx.x / CB;
        L = blockDim.x / CB;
        build_line_twiddles(tw, n);
    }
    __device__ __forceinline__ void swap() {
        double2* t = a;
        a = b;
        b = t;
    }
};

// Transform of the line in t.a, result in t.a (plain plans).
template <bool INV>
__device__ __forceinline__ void line_fft_plain(Tile& t, const SmoothPlan& pl, int CB, bool live) {
    const int c = t.c;
    int Ns = 1;
    for (int s = 0; s < pl.ns; ++s) {
        const int R = pl.r[s];
        const double2* src = t.a;
        double2* dst = t.b;
        if (live) {
            if (R > 16)
                stage_prime<INV>(R, pl.n, Ns, t.lane, t.L, CB, c, t.tw, src, dst);
            else
                with_radix(R, [&](auto rc) {
                    stage<decltype(rc)::value, INV>(pl.n, Ns, t.lane, t.L, t.tw, [&](int i) { return src[i * CB + c]; },
                                                    [&](int i, double2 v) { dst[i * CB + c] = v; });
                });
        }
        __syncthreads();
        t.swap();
        Ns *= R;
    }
}

// Forward or inverse transform of a tile: ld(i) gives point i of the thread's
// channel, st(i, v) takes the result.  REV runs the radices backwards.
template <bool INV, bool REV, class LD, class ST>
__device__ __forceinline__ void line_fft(Tile& t, const SmoothPlan& pl, int CB, bool live, LD&& ld, ST&& st) {
    const int n = pl.n, c = t.c;
    if (pl.plain) {
        if (live)
            for (int i = t.lane; i < n; i += t.L) t.a[i * CB + c] = ld(i);
        __syncthreads();
        line_fft_plain<INV>(t, pl, CB, live);
        if (live)
            for (int i = t.lane; i < n; i += t.L) st(i, t.a[i * CB + c]);
        __syncthreads();
        return;
    }
    int Ns = 1;
    for (int s = 0; s < pl.ns; ++s) {
        const int R = pl.r[REV ? pl.ns - 1 - s : s];
        double2 *src = t.a, *dst = t.b;
        if (live) {
            with_radix(R, [&](auto rc) {
                constexpr int RR = decltype(rc)::value;
                if (s == 0)
                    stage<RR, INV>(n, Ns, t.lane, t.L, t.tw, ld, [&](int i, double2 v) { dst[i * CB + c] = v; });
                else if (s + 1 < pl.ns)
                    stage<RR, INV>(n, Ns, t.lane, t.L, t.tw, [&](int i) { return src[i * CB + c]; },
                                   [&](int i, double2 v) { dst[i * CB + c] = v; });
                else
                    stage<RR, INV>(n, Ns, t.lane, t.L, t.tw, [&](int i) { return src[i * CB + c]; }, st);
            });
        }
        __syncthreads();
        t.swap();
        Ns *= R;
    }
}

// pass A: rows kx < s0 of P (- refP), FFT along ky -> T (s0, n1, Ct)
__global__ void __launch_bounds__(kSmoothThreads, 2)
    k_rows_fwd_m(const double2* __restrict__ P, const double2* __restrict__ refP, double2* T, ExchangeGeom g,
                 SmoothPlan pl, int CB, int nchunk, int ntiles) {
    extern __shared__ __align__(16) unsigned char raw[];
    Tile t(raw, pl.n, CB);
    const size_t nb2 = (size_t)g.nb * g.nb;
    __syncthreads();
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int kx = tile / nchunk, ch = (tile - kx * nchunk) * CB + t.c;
        const bool live = t.lane < t.L && ch < g.C;
        int off = ch;
        if (g.hcp && live) {
            int r = 0, cc = ch;
            while (cc >= g.nb - r) {
                cc -= g.nb - r;
                ++r;
            }
            off = r * g.nb + r + cc;
        }
        const double2* p = P + (size_t)kx * g.s1 * nb2 + off;
        const double2* rp = refP ? refP + (size_t)kx * g.s1 * nb2 + off : nullptr;
        double2* d = T + (size_t)kx * g.n1 * g.Ct + ch;
        line_fft<false, false>(
            t, pl, CB, live,
            [&](int i) {
                if (i >= g.s1) return mk(0.0, 0.0);
                const double2 v = ld_stream(p + (size_t)i * nb2);
                return rp ? csub(v, ld_stream(rp + (size_t)i * nb2)) : v;
            },
            [&](int i, double2 v) { st_l2(d + (size_t)i * g.Ct, v); });
    }
}

// pass B: columns, FFT along kx, * VR (or conj VR), inverse FFT along kx, in place
__global__ void __launch_bounds__(kSmoothThreads, 2)
    k_cols_conv_m(double2* T, const double2* __restrict__ VR, ExchangeGeom g, SmoothPlan pl, int CB, int nchunk,
                  int ntiles, int vmode) {
    extern __shared__ __align__(16) unsigned char raw[];
    Tile t(raw, pl.n, CB);
    const int n = pl.n, c = t.c, sh = g.shift ? g.n0 / 2 : 0;
    __syncthreads();
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int ky = tile / nchunk, ch = (tile - ky * nchunk) * CB + c;
        const bool live = t.lane < t.L && ch < g.C;
        double2* p = T + (size_t)ky * g.Ct + ch;
        const size_t row = (size_t)g.n1 * g.Ct;
        const double2* vp = VR + (size_t)ky * g.dv + (g.dv == 1 ? 0 : ch);
        const size_t vrow = (size_t)g.n1 * g.dv;
        if (pl.plain) {
            if (live)
                for (int i = t.lane; i < n; i += t.L) t.a[i * CB + c] = i < g.s0 ? ld_l2(p + i * row) : mk(0.0, 0.0);
            __syncthreads();
            line_fft_plain<false>(t, pl, CB, live);
            if (vmode == kSmoothForwardOnly) {
                if (live)
                    for (int i = t.lane; i < n; i += t.L) st_l2(p + i * row, t.a[i * CB + c]);
                __syncthreads();
                continue;
            }
            if (live)
                for (int i = t.lane; i < n; i += t.L) {
                    const double2 w = ld_stream(vp + i * vrow), x = t.a[i * CB + c];
                    t.a[i * CB + c] = vmode == kSmoothConjVR ? cmulc(x, w) : cmul(x, w);
                }
            __syncthreads();
            line_fft_plain<true>(t, pl, CB, live);
            if (live)
                for (int i = t.lane; i < n; i += t.L) {
                    const int dx = i >= sh ? i - sh : i - sh + n;
                    if (dx < g.s0) st_l2(p + dx * row, t.a[i * CB + c]);
                }
            __syncthreads();
            continue;
        }
        int Ns = 1;
        // forward stages but the last one
        for (int s = 0; s + 1 < pl.ns; ++s) {
            double2 *src = t.a, *dst = t.b;
            if (live) {
                with_radix(pl.r[s], [&](auto rc) {
                    constexpr int RR = decltype(rc)::value;
                    auto st = [&](int i, double2 v) { dst[i * CB + c] = v; };
                    if (s == 0)
                        stage<RR, false>(n, Ns, t.lane, t.L, t.tw,
                                         [&](int i) { return i < g.s0 ? ld_l2(p + i * row) : mk(0.0, 0.0); }, st);
                    else
                        stage<RR, false>(n, Ns, t.lane, t.L, t.tw, [&](int i) { return src[i * CB + c]; }, st);
                });
            }
            __syncthreads();
            t.swap();
            Ns *= pl.r[s];
        }
        {
            // last forward stage, VR, first inverse stage: butterfly j holds the points
            // j + m n / R before and after the product
            double2 *src = t.a, *dst = t.b;
            if (live) {
                with_radix(pl.r[pl.ns - 1], [&](auto rc) {
                    constexpr int RR = decltype(rc)::value;
                    const int nr = n / RR;
                    for (int j = t.lane; j < nr; j += t.L) {
                        double2 x[RR];
#pragma unroll
                        for (int i = 0; i < RR; ++i) x[i] = src[(j + i * nr) * CB + c];
#pragma unroll
                        for (int i = 1; i < RR; ++i) x[i] = cmul(x[i], t.tw[i * j]);
                        dft_any<RR, false>(x);
                        if (vmode == kSmoothForwardOnly) {
#pragma unroll
                            for (int i = 0; i < RR; ++i) st_l2(p + (j + i * nr) * row, x[i]);
                        } else {
#pragma unroll
                            for (int i = 0; i < RR; ++i) {
                                const double2 w = ld_stream(vp + (j + i * nr) * vrow);
                                x[i] = vmode == kSmoothConjVR ? cmulc(x[i], w) : cmul(x[i], w);
                            }
                            dft_any<RR, true>(x);
#pragma unroll
                            for (int i = 0; i < RR; ++i) dst[(j * RR + i) * CB + c] = x[i];
                        }
                    }
                });
            }
            __syncthreads();
            t.swap();
        }
        if (vmode == kSmoothForwardOnly) continue;
        Ns = pl.r[pl.ns - 1];
        for (int s = pl.ns - 2; s >= 0; --s) {
            double2 *src = t.a, *dst = t.b;
            if (live) {
                with_radix(pl.r[s], [&](auto rc) {
                    constexpr int RR = decltype(rc)::value;
                    auto ld = [&](int i) { return src[i * CB + c]; };
                    if (s > 0)
                        stage<RR, true>(n, Ns, t.lane, t.L, t.tw, ld, [&](int i, double2 v) { dst[i * CB + c] = v; });
                    else
                        stage<RR, true>(n, Ns, t.lane, t.L, t.tw, ld, [&](int i, double2 v) {
                            const int dx = i >= sh ? i - sh : i - sh + n;
                            if (dx < g.s0) st_l2(p + dx * row, v);
                        });
                });
            }
            __syncthreads();
            t.swap();
            Ns *= pl.r[s];
        }
    }
}

// pass C: rows kx < s0 of T, inverse FFT along ky, * scale -> Sigma (s0, s1, nb^2)
__global__ void __launch_bounds__(kSmoothThreads, 2)
    k_rows_inv_m(const double2* T, double2* Sigma, ExchangeGeom g, SmoothPlan pl, int CB, int nchunk, int ntiles,
                 double scale) {
    extern __shared__ __align__(16) unsigned char raw[];
    Tile t(raw, pl.n, CB);
    const size_t nb2 = (size_t)g.nb * g.nb;
    const int sh = g.shift ? g.n1 / 2 : 0;
    __syncthreads();
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int kx = tile / nchunk, ch = (tile - kx * nchunk) * CB + t.c;
        const bool live = t.lane < t.L && ch < g.C;
        int off = ch, mir = -1;
        if (g.hcp && live) {
            int r = 0, cc = ch;
            while (cc >= g.nb - r) {
                cc -= g.nb - r;
                ++r;
            }
            off = r * g.nb + r + cc;
            if (cc > 0) mir = (r + cc) * g.nb + r;
        }
        const double2* p = T + (size_t)kx * g.n1 * g.Ct + ch;
        double2* d = Sigma + (size_t)kx * g.s1 * nb2;
        line_fft<true, true>(
            t, pl, CB, live, [&](int i) { return ld_l2(p + (size_t)i * g.Ct); },
            [&](int i, double2 v) {
                const int dy = i >= sh ? i - sh : i - sh + g.n1;
                if (dy >= g.s1) return;
                v = cscale(v, scale);
                d[(size_t)dy * nb2 + off] = v;
                if (mir >= 0) d[(size_t)dy * nb2 + mir] = cconj(v);
            });
    }
}

// ---------------------------------------------------------------------------
// plans and launches
// ---------------------------------------------------------------------------
// relative cost of a stage per point: shared-memory and twiddle traffic plus the butterfly
double radix_cost(int r) {
    switch (r) {
        case 2: return 9.0;
        case 3: return 10.0;
        case 4: return 10.0;
        case 5: return 12.0;
        case 6: return 11.3;
        case 7: return 14.0;
        case 8: return 11.5;
        case 9: return 12.5;
        case 10: return 13.0;
        case 11: return 18.0;
        case 12: return 12.5;
        case 13: return 20.0;
        case 14: return 15.0;
        case 15: return 14.5;
        default: return 13.0;  // 16
    }
}

// cheapest factorisation of m into at most `depth` radices >= lowest
double factor(int m, int lowest, int depth, int* r, int& ns) {
    if (m == 1) {
        ns = 0;
        return 0.0;
    }
    double best = -1.0;
    if (depth == 0) return best;
    for (int q = lowest; q <= 16; ++q) {
        if (m % q) continue;
        int sub[kSmoothMaxStages], k = 0;
        const double rest = factor(m / q, q, depth - 1, sub, k);
        if (rest < 0.0) continue;
        const double c = radix_cost(q) + rest;
        if (best < 0.0 || c < best) {
            best = c;
            r[0] = q;
            for (int i = 0; i < k; ++i) r[1 + i] = sub[i];
            ns = k + 1;
        }
    }
    return best;
}

bool smooth_plan(int n, SmoothPlan& pl) {
    pl.n = n;
    pl.ns = 0;
    int m = n;
    for (int p : {2, 3, 5, 7, 11, 13})
        while (m % p == 0) m /= p;
    const int smooth = n / m;
    for (int p = 17; m > 1; p += 2) {  // the large primes first: their stages then have no twiddles forward
        if (p * p > m) p = m;
        while (m % p == 0) {
            if (pl.ns == kSmoothMaxStages) return false;
            pl.r[pl.ns++] = p;
            m /= p;
        }
    }
    int k = 0;
    bool ok = smooth == 1;
    for (int d = 1; d <= kSmoothMaxStages - pl.ns && !ok; ++d) ok = factor(smooth, 2, d, pl.r + pl.ns, k) >= 0.0;
    pl.plain = pl.ns > 0 || k < 2;
    pl.ns += k;
    return ok && pl.ns > 0;
}

struct SmoothLaunch {
    int CB, nchunk, threads;
    size_t smem;
};

// channels per tile: about kSmoothTile points (so that two to three CTAs fit an
// SM), fewer (down to four, a 64-byte run) where the pass would have a tile for less than
// three SMs in five, in balanced chunks: 37 x 37, nb = 8 24.2 -> 19.8 us an exchange,
// 19 x 19, nb = 16 29.7 -> 18.1; a tile for every SM instead took 26.9 -> 32.9 at
// 31 x 31, nb = 16
SmoothLaunch smooth_launch(int n, int C, int lines) {
    SmoothLaunch L;
    const int64_t tiles = std::max(1, 3 * num_sms() / 5);
    const int per_sm = (int)std::min<int64_t>(C, ((int64_t)lines * C + tiles - 1) / tiles);
    const int cap = std::max(1, std::min({C, kSmoothTile / n, kSmoothThreads, std::max(per_sm, 4)}));
    const int nch = (C + cap - 1) / cap;
    L.CB = (C + nch - 1) / nch;
    L.nchunk = (C + L.CB - 1) / L.CB;
    L.threads = (kSmoothThreads / L.CB * L.CB + 31) / 32 * 32;
    L.smem = sizeof(double2) * ((size_t)n + 2 * (size_t)n * L.CB);
    return L;
}

template <class K>
int smooth_grid(K kern, const SmoothLaunch& L, int64_t ntiles) {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, L.threads, L.smem);
    (void)cudaGetLastError();
    return (int)std::max<int64_t>(1, std::min<int64_t>(ntiles, (int64_t)std::max(per, 1) * num_sms()));
}

void smooth_attrs() {
    static std::once_flag once;
    std::call_once(once, [] {
        raise_smem(k_rows_fwd_m);
        raise_smem(k_cols_conv_m);
        raise_smem(k_rows_inv_m);
    });
}

bool ready(int n, int C, int lines, SmoothPlan& pl, SmoothLaunch& L) {
    if (!smooth_plan(n, pl)) return false;
    L = smooth_launch(n, C, lines);
    if (L.smem > kSmemMax) return false;
    smooth_attrs();
    return true;
}

}  // namespace

// Small passes wait for the chain of one butterfly, which grows with the radix; the
// Stockham stages of fft.cuh, an output per thread, have the shorter one and lose once
// their R loads and FMAs per point fill the SMs.  Measured in whole exchanges, both row
// passes / the columns pass here less there, us: n = 100 +3.7 / -0.6 up to 2^12 points
// (n x lines x channels), +1.3 / -1.9 in [2^15, 2^16), -2.4 / -5.9 beyond; n = 13 +2.4 /
// +1.2, +1.3 / +0.6, -0.6 / -0.8; n = 21 +0.7 / -1.0, -1.0 / -2.1; n = 75 +3.3 / +0.8,
// +1.1 / -0.6; n = 19 (a direct sum) +0.5 / +0.4 up to 2^13, +0.2 / +0.2, -2.8 / -2.4.
// Longer primes (47: -0.7 / 0; 251: -7.4 / -2.8) and lines of more than 240 points (384:
// -2.9 / -5.8) win or tie here at any size.
bool smooth_pays(int n, int64_t points, bool columns) {
    constexpr int64_t k14 = 1 << 14, k15 = 1 << 15, k16 = 1 << 16;
    SmoothPlan pl;
    if (n > 240 || points >= k16 || !smooth_plan(n, pl)) return true;
    bool long_odd = n < 16 && n % 2 == 1;  // a single radix of 7, 11, 13 or 15 ends in one here
    for (int i = 0; i < pl.ns; ++i) {
        if (pl.r[i] > 16) return n > 37 || points >= k14;
        long_odd = long_odd || pl.r[i] == 13 || pl.r[i] == 15;
    }
    if (columns) return points >= k15 || !long_odd;
    return points >= (n < 16 || (n >= 96 && n <= 192) ? k16 : k15);
}

bool smooth_supported(int n, int C) {
    SmoothPlan pl;
    return smooth_plan(n, pl) && smooth_launch(n, C, 65535).smem <= kSmemMax;
}

int smooth_rows_fwd(const double2* P, const double2* refP, double2* T, const ExchangeGeom& g, cudaStream_t st) {
    SmoothPlan pl;
    SmoothLaunch L;
    if (!ready(g.n1, g.C, g.s0, pl, L)) return fail(CPPHF_ERR_UNSUPPORTED, "exchange: mesh axis too long for the shared-memory FFT");
    const int nt = g.s0 * L.nchunk;
    k_rows_fwd_m<<<smooth_grid(k_rows_fwd_m, L, nt), L.threads, L.smem, st>>>(P, refP, T, g, pl, L.CB, L.nchunk, nt);
    CPPHF_LAUNCH_CHECK("exchange rows forward");
    return CPPHF_OK;
}

int smooth_cols(double2* T, const double2* VR, const ExchangeGeom& g, int vmode, cudaStream_t st) {
    SmoothPlan pl;
    SmoothLaunch L;
    if (!ready(g.n0, g.C, g.n1, pl, L)) return fail(CPPHF_ERR_UNSUPPORTED, "exchange: mesh axis too long for the shared-memory FFT");
    const int nt = g.n1 * L.nchunk;
    k_cols_conv_m<<<smooth_grid(k_cols_conv_m, L, nt), L.threads, L.smem, st>>>(T, VR, g, pl, L.CB, L.nchunk, nt, vmode);
    CPPHF_LAUNCH_CHECK("exchange columns convolve");
    return CPPHF_OK;
}

int smooth_rows_inv(const double2* T, double2* Sigma, const ExchangeGeom& g, double scale, cudaStream_t st) {
    SmoothPlan pl;
    SmoothLaunch L;
    if (!ready(g.n1, g.C, g.s0, pl, L)) return fail(CPPHF_ERR_UNSUPPORTED, "exchange: mesh axis too long for the shared-memory FFT");
    const int nt = g.s0 * L.nchunk;
    k_rows_inv_m<<<smooth_grid(k_rows_inv_m, L, nt), L.threads, L.smem, st>>>(T, Sigma, g, pl, L.CB, L.nchunk, nt, scale);
    CPPHF_LAUNCH_CHECK("exchange rows inverse");
    return CPPHF_OK;
}

}  // namespace cpphf
