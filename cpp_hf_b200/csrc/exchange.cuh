// Internal interface of the exchange (FFT convolution) kernels.
#pragma once

#include "common.cuh"

namespace cpphf {

struct ExchangeGeom {
    int n0, n1;  // mesh (nk1, nk2)
    int nb;      // orbitals
    int C;       // channels transformed: nb*nb, or nb*(nb+1)/2 with HCP
    int dv;      // VR channel width: 1 (scalar broadcast) or nb*nb (elementwise)
    int Ct;      // channel stride of the intermediate T
    int hcp;     // upper-triangle packing with conjugate mirror on unpack: 1 by rows, 2 by 4 x 4 tiles
    int shift;   // apply ifftshift on (kx, ky) to the output
    int s0, s1;  // stored points of a zero-padded field (n0, n1 unless padded)
    unsigned* err = nullptr;  // device error word for bounded waits
};

// Channel order of the upper-triangle packing: by rows (the triangle row-major), or
// by 4 x 4 tiles (tiles of the upper triangle row-major, 16 channels each, entries
// below the diagonal or beyond nb unused), so that 16 consecutive channels are four
// 64-byte row segments of the matrix and their mirrors four others; by rows every
// mirrored entry is a 16-byte access of its own.  The tiles are for the fused build
// of many bands (fock_mesh.cu).  They pay once a field of nk nb^2 entries is large
// enough that P, T and F do not share the L2, and while few of their entries are
// unused.  Measured, fused build by tiles / unfused by rows (us): 2^22 entries and
// <= 1.3 times the triangle's channels: nb 12 at 192 x 192 184/225, 16 at 144 x 144
// 162/192, 33 at 64 x 64 140/146, 64 at 36 x 36 145/179, 28 at 144 x 144 436/633;
// below, nb 24 at 64 x 64 83/81, 33 at 36 x 36 62/55.  Up to 1.6 times (nb 17, 18,
// 21, 22, 25, 29): 17 at 128 x 128 230/209, 25 at 96 x 96 217/214, but 17 at
// 192 x 192 432/482 and 25 at 144 x 144 428/516.  Beyond: 13 at 192 x 192 290/255.
// Without a codelet along ky: 24 at 144 x 100 339/307, 32 at 100 x 100 410/385.
__host__ __device__ inline int hcp_tiles(int nb) { return (nb + 3) / 4; }
inline int hcp_channels(int mode, int nb) {
    const int t = hcp_tiles(nb);
    return mode == 2 ? 8 * t * (t + 1) : nb * (nb + 1) / 2;
}
// whether the fused build takes a complex128 field of this shape by tiles
bool hcp_tiled(int64_t n0, int64_t n1, int64_t nb);
// channel -> (row, col), row <= col; false for an unused channel
__device__ __forceinline__ bool hcp_pair(int ch, int nb, int hcp, int& i, int& j) {
    const int m = hcp == 2 ? hcp_tiles(nb) : nb;
    int r = 0, c = hcp == 2 ? ch >> 4 : ch;
    while (c >= m - r) {
        c -= m - r;
        ++r;
    }
    i = r;
    j = r + c;
    if (hcp == 2) {
        i = 4 * i + ((ch >> 2) & 3);
        j = 4 * j + (ch & 3);
        return i <= j && j < nb;
    }
    return true;
}

size_t exchange_workspace_bytes(int64_t nk1, int64_t nk2, int64_t nb, int hcp, int precision);

// Sigma = -IFFT2[FFT2(P - refP) * VR]; refP may be null; Sigma may alias P.
int exchange(const double2* P, const double2* refP, const double2* VR, double2* Sigma, int64_t nk1,
             int64_t nk2, int64_t nb, int64_t dv, int hcp, int shift, int precision,
             void* workspace, size_t workspace_bytes, cudaStream_t st);

// The full-channel exchange of a zero-padded field, in place: X holds the s0 x s1
// points of the n0 x n1 mesh that are not zero (and receives Sigma at those
// points), T is scratch of s0 * n1 * nb^2 elements.
bool exchange_padded_supported(int64_t n0, int64_t n1, int64_t nb);
int exchange_padded(double2* X, const double2* VR, double2* T, int64_t n0, int64_t n1, int64_t s0, int64_t s1,
                    int64_t nb, int64_t dv, cudaStream_t st);

// The first two passes of the upper-triangle exchange (complex128): T[k, ch] holds,
// along kx, the convolved field, along ky still its transform.
int exchange_hcp_two_passes(const double2* P, const double2* refP, const double2* VR, double2* T, const ExchangeGeom& g,
                            cudaStream_t st);

// The columns pass alone on an (n0, n1, g.C) field T (complex128, or complex64
// with precision 32): FFT along kx, times VR (g.dv = 1: one scalar per q,
// else g.dv = g.C channels laid out like T), inverse FFT along kx, in place.
int exchange_columns(void* T, const double2* VR, const ExchangeGeom& g, int precision, cudaStream_t st);

}  // namespace cpphf
