// Mixed-radix exchange passes (exchange_smooth.cu): complex128, any line length
// that fits shared memory (n <= 4800), optionally zero-padded fields (g.s0 x g.s1 stored points of the n0 x n1 mesh).
#pragma once

#include "exchange.cuh"

namespace cpphf {

// column-pass modes, as in exchange.cu
constexpr int kSmoothVR = 0;
constexpr int kSmoothConjVR = 1;
constexpr int kSmoothForwardOnly = 2;

bool smooth_supported(int n, int C);
// whether a row or columns pass of `points` = n x lines x channels, not padded, is faster here than in fft.cuh's stages
bool smooth_pays(int n, int64_t points, bool columns);
int smooth_rows_fwd(const double2* P, const double2* refP, double2* T, const ExchangeGeom& g, cudaStream_t st);
int smooth_cols(double2* T, const double2* VR, const ExchangeGeom& g, int vmode, cudaStream_t st);
int smooth_rows_inv(const double2* T, double2* Sigma, const ExchangeGeom& g, double scale, cudaStream_t st);

}  // namespace cpphf
