// Recombinations of block vectors x[row * nb + r] with coefficients per right-hand side (blockcombine.cu).
#pragma once
#include "momed_internal.cuh"

namespace momed {

// out[i][n][r] = sum_a U[i][a][r] V[a][n][r] for i < nout (U real, [(i m + a) nb + r]), and out[nout] =
// V[copy_col] when copy_col >= 0.  Sums in FP32 from FP32 to FP32 vectors, else in FP64; out must not
// overlap V.  buf holds the coefficients on the device.
template <typename VIN, typename VOUT>
void block_combine(const VIN* V, int64_t N, int nb, int m, const std::vector<double>& U, int nout, VOUT* out,
                   int copy_col, DevBuf<double>& buf, cudaStream_t st);

// out[i][n][r] = sum_{a<kx} Y[i][a][r] X[a][n][r] + sum_{b<kz} Y[i][kx+b][r] Z[b][n][r]
//               + sum_{j<p} Y[i][kx+kz+j][r] Q[j][n][r]
// for i < nout (Y complex, [(i (kx + kz + p) + a) nb + r]).  FP64 sums; the FP32 source Q in FP32
// arithmetic (its values carry FP32 rounding already), added to the FP64 sums.  out overlaps no source.
void block_combine_c(const double2* X, int kx, const double2* Z, int kz, const float2* Q, int p, int64_t N, int nb,
                     const std::vector<double2>& Y, int nout, double2* out, DevBuf<double2>& buf, cudaStream_t st);

}  // namespace momed
