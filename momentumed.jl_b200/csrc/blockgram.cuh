// Inner products of block vectors x[row * nb + r], per right-hand side r (blockgram.cu).
#pragma once
#include "momed_internal.cuh"

namespace momed {

constexpr int kGramRhs = 4;

// out[(j ncols + i) nb + r] = sum_n conj(V_i[n][r]) R_j[n][r] for i < ncols, j < nr <= kGramRhs, in FP64 and
// in a fixed order.  part: block_gram_part(nb, ncols) values.
size_t block_gram_part(int nb, int ncols);
template <typename VT>
void block_gram(const VT* V, int64_t N, int nb, int ncols, const double2* const* R, int nr, double2* part, double2* out,
                cudaStream_t st);

}  // namespace momed
