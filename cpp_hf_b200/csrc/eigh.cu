// Batched Hermitian eigendecomposition entry points (cpp_hf linalg.hpp:20-140)
// and the off-block norms of the block-diagonal path.  The solvers are
// eigh_small.cu (2 <= nb <= 8, no block structure) and eigh_dc.cu (any nb).
#include "common.cuh"
#include "eigh.cuh"

#include <cstring>

#include <algorithm>
#include <string>
#include <vector>

namespace cpphf {

namespace {

// max |M_ij| over the off-block entries of every matrix (linalg.hpp:123-140).
__global__ void k_max_offblock(const double2* __restrict__ M, int64_t batch, int nb, BlockSpec bs,
                               unsigned long long* out) {
    const int64_t n = batch * (int64_t)nb * nb;
    double m = 0.0;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e % ((int64_t)nb * nb));
        const int i = r / nb, j = r - i * nb;
        if (bs.blk[i] != bs.blk[j]) {
            const double2 a = M[e];
            m = fmax(m, hypot(a.x, a.y));
        }
    }
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// max |M| (out[0]) and max |M_ij| over the off-block entries (out[1]) of a
// batch, as doubles reinterpreted for atomicMax (non-negative, so the integer
// order is the numeric order).
__global__ void k_block_norms(const double2* __restrict__ M, int64_t batch, int nb, BlockSpec bs,
                              unsigned long long* out) {
    const int64_t n = batch * (int64_t)nb * nb;
    double all = 0.0, off = 0.0;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e % ((int64_t)nb * nb));
        const int i = r / nb, j = r - i * nb;
        const double2 a = M[e];
        const double v = hypot(a.x, a.y);
        all = fmax(all, v);
        if (bs.blk[i] != bs.blk[j]) off = fmax(off, v);
    }
    all = warp_max(all);
    off = warp_max(off);
    if ((threadIdx.x & 31) == 0) {
        if (all > 0.0) atomicMax(&out[0], (unsigned long long)__double_as_longlong(all));
        if (off > 0.0) atomicMax(&out[1], (unsigned long long)__double_as_longlong(off));
    }
}

}  // namespace

int eigh_batched(const double2* M, double* w, double2* V, int64_t batch, int64_t nb, int mode,
                 const BlockSpec* bs_in, cudaStream_t st) {
    if (nb < 1 || batch < 0) return fail(CPPHF_ERR_INVALID, "eigh: invalid shape");
    if (batch == 0) return CPPHF_OK;
    if (nb > kMaxEighNb)
        return fail(CPPHF_ERR_UNSUPPORTED, "eigh: nb > " + std::to_string(kMaxEighNb) + " not supported");
    BlockSpec bs;
    if (bs_in)
        bs = *bs_in;
    else {
        bs.nblocks = 1;
        bs.sort = 1;
        bs.start[0] = 0;
        bs.start[1] = (short)nb;
        for (int i = 0; i < nb; ++i) bs.blk[i] = 0;
    }
    if (bs.nblocks <= 1 && eigh_small_enabled(nb)) return eigh_small(M, w, V, batch, nb, mode, st);
    if (eigh_blocks_enabled(batch, bs)) return eigh_blocks(M, w, V, batch, nb, mode, bs, st);
    return eigh_dc(M, w, V, batch, nb, mode, bs, st);
}

int block_structure_ok(const double2* M, int64_t batch, int64_t nb, const BlockSpec& bs, unsigned long long* dev2,
                       cudaStream_t st, bool* ok) {
    *ok = true;
    if (batch <= 0) return CPPHF_OK;
    CPPHF_CUDA(cudaMemsetAsync(dev2, 0, 2 * sizeof(unsigned long long), st));
    const int64_t n = batch * nb * nb;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 8));
    k_block_norms<<<grid, 256, 0, st>>>(M, batch, (int)nb, bs, dev2);
    CPPHF_LAUNCH_CHECK("block structure check");
    unsigned long long h[2] = {0ull, 0ull};
    CPPHF_CUDA(cudaMemcpyAsync(h, dev2, sizeof(h), cudaMemcpyDeviceToHost, st));
    CPPHF_CUDA(cudaStreamSynchronize(st));
    double scale, off;
    std::memcpy(&scale, &h[0], sizeof(double));
    std::memcpy(&off, &h[1], sizeof(double));
    *ok = off <= 1.0e-10 + 1.0e-10 * scale;
    return CPPHF_OK;
}

int make_block_spec(int64_t nb, const int64_t* sizes, int64_t n_sizes, int sort, BlockSpec& bs) {
    if (n_sizes < 1 || n_sizes > kMaxEighNb) return fail(CPPHF_ERR_INVALID, "block sizes must sum to nb");
    int64_t tot = 0;
    for (int64_t b = 0; b < n_sizes; ++b) {
        if (sizes[b] <= 0) return fail(CPPHF_ERR_INVALID, "block_sizes entries must be positive.");
        tot += sizes[b];
    }
    if (tot != nb) return fail(CPPHF_ERR_INVALID, "block sizes must sum to nb");
    bs.nblocks = (int)n_sizes;
    bs.sort = sort ? 1 : 0;
    int s0 = 0;
    for (int b = 0; b < n_sizes; ++b) {
        bs.start[b] = (short)s0;
        for (int i = 0; i < sizes[b]; ++i) bs.blk[s0 + i] = (unsigned char)b;
        s0 += (int)sizes[b];
    }
    bs.start[n_sizes] = (short)s0;
    return CPPHF_OK;
}

}  // namespace cpphf

extern "C" {

int cpphf_eigh_batched(const void* M, double* w, void* V, int64_t batch, int64_t nb, void* stream) {
    return cpphf::eigh_batched(static_cast<const double2*>(M), w, static_cast<double2*>(V), batch, nb,
                               0, nullptr, static_cast<cudaStream_t>(stream));
}

int cpphf_eigh_block_sizes(const void* M, double* w, void* V, int64_t batch, int64_t nb,
                           const int64_t* sizes, int64_t n_sizes, int sort, void* stream) {
    cpphf::BlockSpec bs;
    CPPHF_TRY(cpphf::make_block_spec(nb, sizes, n_sizes, sort, bs));
    return cpphf::eigh_batched(static_cast<const double2*>(M), w, static_cast<double2*>(V), batch, nb,
                               0, &bs, static_cast<cudaStream_t>(stream));
}


int cpphf_max_offblock_sizes(const void* M, int64_t batch, int64_t nb, const int64_t* sizes, int64_t n_sizes,
                             double* out, void* stream) {
    cpphf::BlockSpec bs;
    int64_t tot = 0;
    for (int64_t b = 0; b < n_sizes; ++b) tot += sizes[b];
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    CPPHF_CUDA(cudaMemsetAsync(out, 0, sizeof(double), st));
    if (nb > cpphf::kMaxEighNb || n_sizes < 1 || tot != nb || batch <= 0) {
        // linalg.hpp:123-140 tolerates any sizes; only the covered region is masked
        if (nb > cpphf::kMaxEighNb) return cpphf::fail(CPPHF_ERR_UNSUPPORTED, "max_offblock_sizes: nb too large");
        if (batch <= 0) return CPPHF_OK;
    }
    bs.nblocks = 0;
    bs.sort = 1;
    // entries outside every listed block belong to their own pseudo-block
    for (int i = 0; i < nb; ++i) bs.blk[i] = (unsigned char)(100 + i);  // unique id per uncovered index
    int s0 = 0;
    for (int64_t b = 0; b < n_sizes && b < 100; ++b) {
        for (int64_t i = 0; i < sizes[b] && s0 + i < nb; ++i) bs.blk[s0 + i] = (unsigned char)b;
        s0 += (int)sizes[b];
    }
    const int64_t n = batch * nb * nb;
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 4096));
    cpphf::k_max_offblock<<<grid, 256, 0, st>>>(static_cast<const double2*>(M), batch, (int)nb, bs,
                                                reinterpret_cast<unsigned long long*>(out));
    CPPHF_LAUNCH_CHECK("max_offblock");
    return CPPHF_OK;
}

int cpphf_cayley_spectral_setup(const void* d, void* V, double* lam, int64_t batch, int64_t nb,
                                void* stream) {
    return cpphf::eigh_batched(static_cast<const double2*>(d), lam, static_cast<double2*>(V), batch,
                               nb, 1, nullptr, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
