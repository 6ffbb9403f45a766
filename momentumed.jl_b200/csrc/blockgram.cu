// Gram blocks of the lockstep solver's Rayleigh-Ritz: columns of V against up to four right-hand sides.
//
// A block runs through a contiguous range of values, 64 at a time: the values of up to 32 columns and of
// the right-hand sides come through a ring in shared memory (cp.async), a warp takes up to four of the
// columns against all right-hand sides, so each value of V serves four products and each value of a
// right-hand side four, and is converted to FP64 once for them.  A lane keeps to one r (64 is a multiple
// of nb), so only the sums cross lanes, once per block.
//
// What bounds it: HBM, and the FP64 products beside the shared-memory reads of the right-hand sides.  On
// 173.6k states x 32 (B200): 8 FP64 columns against 4 right-hand sides 174 us (1.07 GB, 6.1 TB/s), 22 c64
// columns 301 us (1.3 GB; 0.11 ms of FP64 products), where a warp per column with the right-hand sides
// through L1 took 245 and 860 us, and one right-hand side at a time 270 us each.
#include <algorithm>
#include <type_traits>

#include "blockgram.cuh"
#include "packets.cuh"

namespace momed {

namespace {

constexpr int kT = 256;
constexpr int kVals = 64;              // values of a stage
constexpr int kCols = 32;              // columns of a pass: four for each warp
constexpr unsigned kAll = 0xffffffffu;

template <typename VT> constexpr int gram_stages() { return sizeof(VT) == 8 ? 5 : 3; }
template <typename VT> constexpr size_t gram_stage() { return kVals * (kCols * sizeof(VT) + kGramRhs * sizeof(double2)); }

struct Rhs {
    const double2* p[kGramRhs];
};

template <typename VT>
__global__ void __launch_bounds__(kT, 2)
k_block_gram(const VT* __restrict__ V, int64_t total, int nb, int ncols, Rhs R, int nr, double2* __restrict__ part) {
    constexpr int S = gram_stages<VT>();
    extern __shared__ __align__(16) unsigned char sm[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int y = blockIdx.y, ny = gridDim.y;
    const int c0 = (int)((int64_t)y * ncols / ny), cn = (int)((int64_t)(y + 1) * ncols / ny) - c0;   // this pass
    const int w0 = wid * cn / 8, cnt = (wid + 1) * cn / 8 - w0;                                      // this warp
    const int64_t ns = (total + kVals - 1) / kVals;
    const int64_t s0 = ns * blockIdx.x / gridDim.x, s1 = ns * (blockIdx.x + 1) / gridDim.x;
    auto rhs_at = [&](int s) { return reinterpret_cast<double2*>(sm + s * gram_stage<VT>()); };
    auto col_at = [&](int s) { return reinterpret_cast<VT*>(sm + s * gram_stage<VT>() + kGramRhs * kVals * sizeof(double2)); };
    auto fetch = [&](int64_t st, int slot) {
        if (st < s1) {
            const int x = threadIdx.x % kVals, g = threadIdx.x / kVals;
            const int64_t e = st * kVals + x;
            double2* rd = rhs_at(slot) + g * kVals + x;
            VT* cd = col_at(slot) + g * kVals + x;
            const VT* v = V + (int64_t)(c0 + g) * total + e;
            if (e < total) {
                copy_packet(rd, R.p[g] + e);
                for (int c = g; c < cn; c += kT / kVals, cd += kT, v += (kT / kVals) * total) copy_packet(cd, v);
            } else {                               // past the end: zeros
                *rd = make_double2(0.0, 0.0);
                for (int c = g; c < cn; c += kT / kVals, cd += kT) {
                    cd->x = 0;
                    cd->y = 0;
                }
            }
        }
        copy_commit();
    };
    double ax[4][kGramRhs], ay[4][kGramRhs];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int j = 0; j < kGramRhs; ++j) ax[c][j] = ay[c][j] = 0.0;
    auto run = [&](auto CNT) {                     // the warp's count of columns fixed
        constexpr int C = decltype(CNT)::value;
        int slot = 0, next = S - 1;
#pragma unroll
        for (int k = 0; k < S - 1; ++k) fetch(s0 + k, k);
        for (int64_t st = s0; st < s1; ++st) {
            copy_wait<S - 2>();
            __syncthreads();                       // the stage is complete, and the one before is read by all
            fetch(st + S - 1, next);
            next = next == S - 1 ? 0 : next + 1;
            const double2* rp = rhs_at(slot) + lane;
            const VT* vp = col_at(slot) + w0 * kVals + lane;
            slot = slot == S - 1 ? 0 : slot + 1;
#pragma unroll
            for (int k = 0; k < kVals; k += 32) {
                double2 w[kGramRhs];
#pragma unroll
                for (int j = 0; j < kGramRhs; ++j) w[j] = rp[j * kVals + k];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const VT t = vp[c * kVals + k];
                    const double vx = t.x, vy = t.y;
#pragma unroll
                    for (int j = 0; j < kGramRhs; ++j) {
                        ax[c][j] = fma(vx, w[j].x, ax[c][j]);
                        ay[c][j] = fma(vx, w[j].y, ay[c][j]);
                    }
#pragma unroll
                    for (int j = 0; j < kGramRhs; ++j) {
                        ax[c][j] = fma(vy, w[j].y, ax[c][j]);
                        ay[c][j] = fma(-vy, w[j].x, ay[c][j]);
                    }
                }
            }
        }
    };
    switch (cnt) {                                 // all branches meet the same number of barriers
        case 0: run(std::integral_constant<int, 0>{}); break;
        case 1: run(std::integral_constant<int, 1>{}); break;
        case 2: run(std::integral_constant<int, 2>{}); break;
        case 3: run(std::integral_constant<int, 3>{}); break;
        default: run(std::integral_constant<int, 4>{}); break;
    }
    copy_wait<0>();
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (c < cnt) {                             // warp-uniform
#pragma unroll
            for (int j = 0; j < kGramRhs; ++j) {
                double sx = ax[c][j], sy = ay[c][j];
                for (int o = nb; o < 32; o <<= 1) {
                    sx += __shfl_xor_sync(kAll, sx, o);
                    sy += __shfl_xor_sync(kAll, sy, o);
                }
                if (j < nr && lane < nb)
                    part[(((int64_t)blockIdx.x * nr + j) * ncols + c0 + w0 + c) * nb + lane] = make_double2(sx, sy);
            }
        }
}

// out[e] = sum over blocks b < grid of part[b count + e], one warp per element (fixed order)
__global__ void k_block_gram_sum(const double2* __restrict__ part, int grid, int64_t count, double2* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t e = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (e >= count) return;
    double sx = 0.0, sy = 0.0;
    for (int b = lane; b < grid; b += 32) {
        const double2 v = part[b * count + e];
        sx += v.x;
        sy += v.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(kAll, sx, o);
        sy += __shfl_xor_sync(kAll, sy, o);
    }
    if (lane == 0) out[e] = make_double2(sx, sy);
}

// one wave of resident blocks, two per SM, over the column passes
int gram_blocks(int ncols) {
    static const int sms = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 148;
    }();
    return std::max(1, 2 * sms / ((ncols + kCols - 1) / kCols));
}

}  // namespace

size_t block_gram_part(int nb, int ncols) { return (size_t)gram_blocks(ncols) * kGramRhs * ncols * nb; }

template <typename VT>
void block_gram(const VT* V, int64_t N, int nb, int ncols, const double2* const* R, int nr, double2* part, double2* out,
                cudaStream_t st) {
    const int64_t total = N * nb;
    const int rb = (int)std::min<int64_t>(gram_blocks(ncols), (total + kVals - 1) / kVals);
    constexpr int smem = (int)(gram_stages<VT>() * gram_stage<VT>());
    Rhs r{};
    for (int j = 0; j < kGramRhs; ++j) r.p[j] = R[std::min(j, nr - 1)];
    MOMED_CUDA_TRY(cudaFuncSetAttribute(k_block_gram<VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_block_gram<VT><<<dim3(rb, (ncols + kCols - 1) / kCols), kT, smem, st>>>(V, total, nb, ncols, r, nr, part);
    const int64_t count = (int64_t)nr * ncols * nb;
    k_block_gram_sum<<<(unsigned)((count + 7) / 8), 256, 0, st>>>(part, rb, count, out);
    MOMED_CUDA_TRY(cudaGetLastError());
}

template void block_gram<float2>(const float2*, int64_t, int, int, const double2* const*, int, double2*, double2*, cudaStream_t);
template void block_gram<double2>(const double2*, int64_t, int, int, const double2* const*, int, double2*, double2*, cudaStream_t);

}  // namespace momed
