// Fock build of many bands with a scalar V (upper-triangle exchange in 4 x 4 tiles,
// exchange.cuh) with the assembly and the energy fused into the last pass.
//
// Unfused, the last exchange pass writes Sigma (its mirrored entries one by one)
// and the assembly reads it back with h and P to write F.  Here a CTA takes one
// (kx, tile) line at a time: inverse rows transform of the tile's 16 channels, the
// line back into shared memory in natural order, then per (ky, entry) of the tile
//   Sigma += SC, F = herm(h + Sigma + diag(hd)), both (i, j) and (j, i), and the
//   energy terms w_k Re[h_ij P_ji + (Sigma + H)_ij (P - refP)_ji / 2] of the pair,
// all in 64-byte segments of the fields.  Sigma is written only when asked for.
// CTAs are persistent; the energy is Kahan-summed per thread and reduced by the
// last block in a fixed order.
//
// Bound by HBM: T, h and P read, F (and Sigma) written, 4.5 fields of nk nb^2 with
// Sigma.  Measured, 144 x 144, nb = 64 (1.36 GB a field): whole build 2150 us, unfused
// 3920; this pass 1350 us of it (960 at the copy rate).
#include "common.cuh"
#include "exchange.cuh"
#include "exchange_pipe.cuh"
#include "fft_reg.cuh"
#include "fock.cuh"
#include "fock_mesh.cuh"
#include "team.cuh"

#include <algorithm>

namespace cpphf {

namespace {

// A thread per (lane, channel): 256-byte runs of T, 128-byte ones for lines of more
// than 16 lanes.  At least 65536 / 96 resident threads per SM: the assembly waits on its
// loads, and more lines in flight outweigh the spills of the long transforms (144 x 144,
// nb = 64: 2140 us with at most 96 registers, 2330 with 128 or 168, 2330 with 80; two or
// three points loaded ahead per thread, and L2 prefetches of h and P, were slower).
template <int N1, int N2>
struct MeshShape {
    static constexpr int lanes = N1 > N2 ? N1 : N2;
    static constexpr int CB = lanes <= 16 ? 16 : 8;
    static constexpr int threads = (lanes * CB + 31) / 32 * 32;
    static constexpr int ctas = 65536 / (96 * threads);
};

template <int N1, int N2>
__global__ void __launch_bounds__(MeshShape<N1, N2>::threads, MeshShape<N1, N2>::ctas)
    k_rows_inv_mesh(const double2* __restrict__ T, MeshOut o, ExchangeGeom g, int nchunk, int ntiles, double scale) {
    constexpr int N = N1 * N2, CB = MeshShape<N1, N2>::CB, L = MeshShape<N1, N2>::threads / CB;
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ double red[32];
    double2* tw = reinterpret_cast<double2*>(raw);
    double2* S = tw + N;
    const int c = threadIdx.x % CB, a = threadIdx.x / CB;
    build_line_twiddles(tw, N);
    const int nb = g.nb;
    const size_t nb2 = (size_t)nb * nb;
    Kahan e_k;
    __syncthreads();
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int kx = tile / nchunk, ch = (tile - kx * nchunk) * CB + c;
        int i = 0, j = 0;
        const bool live = a < L && hcp_pair(ch, nb, 2, i, j);
        const size_t ij = (size_t)i * nb + j, ji = (size_t)j * nb + i;
        if (a < N1) {
            double2 u[N2];
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) u[k2] = ld_stream(T + ((size_t)kx * N + (a + N1 * k2)) * g.Ct + ch);
            dft<N2, true>(u);
#pragma unroll
            for (int na = 0; na < N2; ++na) S[(a * N2 + na) * CB + c] = cmulc(u[na], tw[na * a]);
        }
        __syncthreads();
        double2 v[N1];
        if (a < N2) {
#pragma unroll
            for (int k1 = 0; k1 < N1; ++k1) v[k1] = S[(k1 * N2 + a) * CB + c];
            dft<N1, true>(v);
        }
        __syncthreads();
        if (a < N2) {
#pragma unroll
            for (int nbx = 0; nbx < N1; ++nbx) S[(a + N2 * nbx) * CB + c] = cscale(v[nbx], scale);
        }
        __syncthreads();
        // thread (a, c) takes the points a, a + L, ... of its own channel: a warp covers
        // whole tile rows of a point
        if (live) {
            const bool diag = i == j;
            const double2 cij = o.SC ? o.SC[ij] : mk(0.0, 0.0), cji = o.SC ? o.SC[ji] : mk(0.0, 0.0);
            const double hd = (diag && o.hd) ? o.hd[i] : 0.0;
#pragma unroll 1
            for (int ky = a; ky < N; ky += L) {
                const size_t k = (size_t)kx * N + ky, at = k * nb2;
                const double2 hij = ld_stream(o.h + at + ij), hji = ld_stream(o.h + at + ji);
                const double2 pij = ld_stream(o.P + at + ij), pji = ld_stream(o.P + at + ji);
                double2 dij = pij, dji = pji;
                if (o.refP) {
                    dij = csub(pij, ld_stream(o.refP + at + ij));
                    dji = csub(pji, ld_stream(o.refP + at + ji));
                }
                const double2 x = S[ky * CB + c];
                const double2 sij = cadd(x, cij), sji = diag ? sij : cadd(cconj(x), cji);
                double2 Aij = cadd(hij, sij), Aji = cadd(hji, sji);
                if (diag) {
                    Aij.x += hd;
                    Aji = Aij;
                }
                const double2 f = mk(0.5 * (Aij.x + Aji.x), 0.5 * (Aij.y - Aji.y));
                __stcs(o.F + at + ij, f);
                if (!diag) __stcs(o.F + at + ji, cconj(f));
                if (o.Sigma) {
                    __stcs(o.Sigma + at + ij, sij);
                    if (!diag) __stcs(o.Sigma + at + ji, sji);
                }
                if (o.Hdense) {
                    o.Hdense[at + ij] = mk(hd, 0.0);
                    if (!diag) o.Hdense[at + ji] = mk(0.0, 0.0);
                }
                double2 iij = cscale(sij, 0.5);
                iij.x += 0.5 * hd;
                double e = (hij.x * pji.x - hij.y * pji.y) + (iij.x * dji.x - iij.y * dji.y);
                if (!diag) {
                    const double2 iji = cscale(sji, 0.5);
                    e += (hji.x * pij.x - hji.y * pij.y) + (iji.x * dij.x - iji.y * dij.y);
                }
                e_k.add(o.w[k] * e);
            }
        }
        __syncthreads();
    }
    if (o.energy) {
        double acc[1] = {e_k.s}, out[1];
        if (reduce_last_block<1>(acc, o.part, o.counter, out, red) && threadIdx.x == 0) *o.energy = out[0];
    }
}

template <int N1, int N2>
int launch(const double2* T, const MeshOut& o, const ExchangeGeom& g, cudaStream_t st) {
    constexpr int N = N1 * N2, CB = MeshShape<N1, N2>::CB, threads = MeshShape<N1, N2>::threads;
    constexpr size_t smem = sizeof(double2) * ((size_t)N + (size_t)N * CB);
    static const int ctas = [] {
        raise_smem(k_rows_inv_mesh<N1, N2>);
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_rows_inv_mesh<N1, N2>, threads, smem);
        (void)cudaGetLastError();
        return std::min(std::max(per, 1) * num_sms(), kFockMaxPartials);
    }();
    const int nchunk = g.C / CB, nt = g.n0 * nchunk;
    if (o.energy) CPPHF_CUDA(cudaMemsetAsync(o.counter, 0, sizeof(unsigned), st));
    k_rows_inv_mesh<N1, N2><<<std::min(nt, ctas), threads, smem, st>>>(T, o, g, nchunk, nt,
                                                                      -1.0 / ((double)g.n0 * (double)g.n1));
    CPPHF_LAUNCH_CHECK("inverse rows with the Fock assembly");
    return CPPHF_OK;
}

}  // namespace

bool fock_mesh_eligible(const cpphf_kernel* K) {
    if (!K->include_exchange || !K->exchange_hcp || K->dv != 1 || K->exchange_precision != 64) return false;
    if (K->sl && (K->sl->fock_active || K->sl->hartree_active)) return false;
    return hcp_tiled(K->nk1, K->nk2, K->nb);
}

size_t fock_mesh_bytes(const cpphf_kernel* K) {
    if (!fock_mesh_eligible(K)) return 0;
    return sizeof(double2) * (size_t)K->nk1 * K->nk2 * hcp_channels(2, (int)K->nb);
}

int build_fock_mesh(const cpphf_kernel* K, const MeshOut& o, void* T, cudaStream_t st) {
    ExchangeGeom g;
    g.n0 = g.s0 = (int)K->nk1;
    g.n1 = g.s1 = (int)K->nk2;
    g.nb = (int)K->nb;
    g.hcp = 2;
    g.C = g.Ct = hcp_channels(2, g.nb);
    g.dv = 1;
    g.shift = 0;
    g.err = wait_error_word();
    if (!g.err) return CPPHF_ERR_CUDA;
    double2* Td = static_cast<double2*>(T);
    CPPHF_TRY(exchange_hcp_two_passes(o.P, o.refP, static_cast<const double2*>(K->VR), Td, g, st));
    switch (g.n1) {
#define X(N, A, B) \
    case N: return launch<A, B>(Td, o, g, st);
        CPPHF_SPEC_SIZES(X)
#undef X
        default: break;
    }
    return fail(CPPHF_ERR_UNSUPPORTED, "build_fock: no codelet for the mesh");
}

}  // namespace cpphf
