// A step of the lockstep block Lanczos beside its map as one cooperative kernel.
//
// The separate kernels of a step (projection, its reduction, update, the test for a second
// Gram-Schmidt pass, that pass, the norms, the scaling: nine launches) cost more than their work on
// sectors of some thousand states, and on large ones the projection converted every value of w to
// FP64 once per column and the update read each coefficient once per packet.  Here a block owns a
// contiguous range of rows for the step and the blocks meet at three grid barriers:
//
//   c[i][r] = V_i[r]^H w[r]     a warp reads up to 8 columns against one read of w; partials per block  | barrier
//   c summed over the blocks    a warp per (column, right-hand side) over the whole grid                | barrier
//   w -= sum c V                two packets of a thread share each coefficient; |w|^2 per block         | barrier
//   (all three once more for the right-hand sides that lost more than the kept share of |w|^2)
//   w /= |w|                    the block's own rows
//
// Every sum is taken in a fixed order, so a solve repeats to the bit.
//
// What bounds it: HBM on large sectors.  Copies run ahead through a ring in shared memory (cp.async, a
// thread waits for its own alone), one block of 256 threads an SM: two blocks an SM, or a deeper ring,
// gained nothing (370 and 379 us against 365).  A step of the 173.6k state sector of a 3x9 mesh with 32
// right-hand sides in c64 (21 columns of 44 MB on average, read twice: 1.9 GB) takes 364 us on the B200
// where the separate kernels took 418, at 6.2 TB/s within a phase; the blocks of an SM that gets less of
// the memory bandwidth finish 20 us after the mean, which both phases wait for.  Without the ring (direct
// loads, two blocks an SM) 441 us; w read once per column group by groups that run apart, 390.  On a
// 5.5k state sector with 16 right-hand sides the step takes 21 us (three barriers of 1.8 us, two phases
// of 5.5) against 34, and the solve 7.8 ms against 11.6, as no graph of small launches is captured.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "blockstep.cuh"
#include "packets.cuh"

namespace momed {

namespace {

constexpr int kBT = 256;               // threads of a block
constexpr int kBW = kBT / 32;
constexpr int kCG = 8;                 // columns of one read of w: 64 registers of FP64 sums for two c64 values
constexpr int kStages = 3;             // ring of the projections: stages of kCG columns and w, 108 KB of 16-byte packets
constexpr int kUpCols = 2, kUpStages = 5;   // ring of the updates: 2 columns of 2 packets, 80 KB beside the coefficients;
                                            // with the coefficients of 135 columns and 32 right-hand sides 149 KB
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ double wred(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
    return v;
}

// part[(c NB + r)][block] for c < ncols (and |w_r|^2 as c = ncols when norm).  The columns are dealt to
// par groups of ch warps; the warps of a group take turns in rows.
template <typename VT, int NB>
__device__ __forceinline__ void step_proj(const BlockStepArgs<VT>& a, int ncols_all, bool norm_all, int64_t r0, int nr,
                                          const VT* w, double2* sm, double* rn) {
    using P = Pack<VT, NB>;
    using PT = typename P::T;
    constexpr int E = P::E, PR = NB / E, RS = 32 / PR;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int rp = lane % PR, rs = lane / PR;
    const int64_t ld = a.N * PR;                              // packets of a column
    constexpr int kStage = (kCG + 1) * kBT;                   // w after the columns
    PT* ring = reinterpret_cast<PT*>(sm) + threadIdx.x;       // [kStages][kCG + 1][kBT]
    double2* red = sm;                                        // [kBW][kCG][NB] after the last copy
    for (int b0 = 0; b0 < ncols_all; b0 += kBW * kCG) {
        const int ncols = min(kBW * kCG, ncols_all - b0);
        const bool norm = norm_all && b0 == 0;
        int par = 1;
        while (par * kCG < ncols) par *= 2;
        const int ch = kBW / par, q = wid % ch, g = wid / ch;
        const int c0 = g * ncols / par, cnt = (g + 1) * ncols / par - c0;   // warp-uniform, at most kCG
        double ax[kCG][E], ay[kCG][E], n2[E];
#pragma unroll
        for (int e = 0; e < E; ++e) n2[e] = 0.0;
#pragma unroll
        for (int c = 0; c < kCG; ++c)
#pragma unroll
            for (int e = 0; e < E; ++e) ax[c][e] = ay[c][e] = 0.0;
        const int step = ch * RS, first = q * RS + rs, its = (nr - q * RS + step - 1) / step;   // warp-uniform
        auto rows = [&](auto CNT) {                           // the count of columns fixed: no test per column
            constexpr int C = decltype(CNT)::value;
            const PT* fw = reinterpret_cast<const PT*>(w) + (r0 + first) * PR + rp;      // the next copy
            const PT* fv = reinterpret_cast<const PT*>(a.V) + (b0 + c0) * ld + (r0 + first) * PR + rp;
            int ft = first, fo = 0, uo = 0;
            auto fetch = [&] {
                if (ft < nr) {
                    PT* d = ring + fo;
                    copy_packet(d + kCG * kBT, fw);
                    const PT* v = fv;
#pragma unroll
                    for (int c = 0; c < C; ++c, v += ld) copy_packet(d + c * kBT, v);
                }
                copy_commit();
                ft += step;
                fw += step * PR;
                fv += step * PR;
                fo = fo == (kStages - 1) * kStage ? 0 : fo + kStage;
            };
#pragma unroll
            for (int k = 0; k < kStages - 1; ++k) fetch();
            for (int it = 0; it < its; ++it) {
                const bool in = ft - (kStages - 1) * step < nr;
                fetch();
                copy_wait<kStages - 1>();
                if (in) {
                    const PT* d = ring + uo;
                    double2 x[E];
                    P::get(d[kCG * kBT], x);
#pragma unroll
                    for (int e = 0; e < E; ++e) n2[e] = fma(x[e].y, x[e].y, fma(x[e].x, x[e].x, n2[e]));
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        double2 y[E];
                        P::get(d[c * kBT], y);
#pragma unroll
                        for (int e = 0; e < E; ++e) {
                            ax[c][e] = fma(y[e].x, x[e].x, ax[c][e]);
                            ay[c][e] = fma(y[e].x, x[e].y, ay[c][e]);
                        }
#pragma unroll
                        for (int e = 0; e < E; ++e) {
                            ax[c][e] = fma(y[e].y, x[e].y, ax[c][e]);
                            ay[c][e] = fma(-y[e].y, x[e].x, ay[c][e]);
                        }
                    }
                }
                uo = uo == (kStages - 1) * kStage ? 0 : uo + kStage;
            }
        };
        switch (cnt) {
            case 1: rows(std::integral_constant<int, 1>{}); break;
            case 2: rows(std::integral_constant<int, 2>{}); break;
            case 3: rows(std::integral_constant<int, 3>{}); break;
            case 4: rows(std::integral_constant<int, 4>{}); break;
            case 5: rows(std::integral_constant<int, 5>{}); break;
            case 6: rows(std::integral_constant<int, 6>{}); break;
            case 7: rows(std::integral_constant<int, 7>{}); break;
            default: rows(std::integral_constant<int, kCG>{}); break;
        }
        copy_wait<0>();
        __syncthreads();                                      // the ring becomes red
#pragma unroll
        for (int c = 0; c < kCG; ++c)
            if (c < cnt) {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    double sx = ax[c][e], sy = ay[c][e];
#pragma unroll
                    for (int o = PR; o < 32; o <<= 1) {
                        sx += __shfl_xor_sync(kAll, sx, o);
                        sy += __shfl_xor_sync(kAll, sy, o);
                    }
                    if (rs == 0) red[(wid * kCG + c) * NB + rp * E + e] = make_double2(sx, sy);
                }
            }
#pragma unroll
        for (int e = 0; e < E; ++e) {
            double s = n2[e];
#pragma unroll
            for (int o = PR; o < 32; o <<= 1) s += __shfl_xor_sync(kAll, s, o);
            if (rs == 0) rn[wid * NB + rp * E + e] = s;       // group 0's warps hold |w|^2 once
        }
        __syncthreads();
        for (int e = threadIdx.x; e < par * kCG * NB; e += kBT) {
            const int gg = e / (kCG * NB), c = e / NB % kCG, r = e % NB;
            const int cb = gg * ncols / par;
            if (c < (gg + 1) * ncols / par - cb) {
                const double2* s = red + (gg * ch * kCG + c) * NB + r;
                double sx = 0.0, sy = 0.0;
                for (int k = 0; k < ch; ++k) { sx += s[k * kCG * NB].x; sy += s[k * kCG * NB].y; }
                a.part[(int64_t)((b0 + cb + c) * NB + r) * gridDim.x + blockIdx.x] = make_double2(sx, sy);
            }
        }
        if (norm && threadIdx.x < NB) {
            double s = 0.0;
            for (int k = 0; k < ch; ++k) s += rn[k * NB + threadIdx.x];
            a.part[(int64_t)(ncols_all * NB + threadIdx.x) * gridDim.x + blockIdx.x] = make_double2(s, 0.0);
        }
        __syncthreads();
    }
}

// coef[e] = sum over the blocks of part[e], a warp of the grid per element
template <typename VT> __device__ __forceinline__ void step_reduce(const BlockStepArgs<VT>& a, int count) {
    const int lane = threadIdx.x & 31;
    for (int e = blockIdx.x * kBW + (threadIdx.x >> 5); e < count; e += gridDim.x * kBW) {
        const double2* p = a.part + (int64_t)e * gridDim.x;
        double sx = 0.0, sy = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) {
            const double2 v = __ldcg(p + b);
            sx += v.x;
            sy += v.y;
        }
        sx = wred(sx);
        sy = wred(sy);
        if (lane == 0) a.coef[e] = make_double2(sx, sy);
    }
}

// w -= sum_i coef[i][r] V_i on the block's rows, |w_r|^2 per block; cs: the coefficients, the packets of
// a row side by side.  A thread takes two packets at a time; its copies run on over the pairs.
template <typename VT, int NB>
__device__ __forceinline__ void step_update(const BlockStepArgs<VT>& a, int ncols, int64_t r0, int nr, VT* w,
                                            double2* sm, const double2* cs, double* rn) {
    using P = Pack<VT, NB>;
    using PT = typename P::T;
    constexpr int E = P::E, PR = NB / E;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int rp = threadIdx.x % PR;
    const int64_t ld = a.N * PR;
    const int total = nr * PR;
    const PT* vp = reinterpret_cast<const PT*>(a.V) + r0 * PR + threadIdx.x;
    PT* wp = reinterpret_cast<PT*>(w) + r0 * PR + threadIdx.x;
    PT* ring = reinterpret_cast<PT*>(sm) + threadIdx.x;       // [kUpStages][kUpCols][2][kBT]
    double n2[E];
#pragma unroll
    for (int e = 0; e < E; ++e) n2[e] = 0.0;
    const int left = total - (int)threadIdx.x;                // packet p of the thread exists when p < left
    const int pairs = (total + 2 * kBT - 1) / (2 * kBT);   // block-uniform
    constexpr int kStage = kUpCols * 2 * kBT;
    int fp = 0, fi = 0, fo = 0;                               // the next copy: pair's first packet, column, stage
    const PT* fv = vp;
    auto fetch = [&] {
        if (fp < left) {
            PT* d = ring + fo;
            const bool both = fp + kBT < left;
            copy_packet(d, fv);
            if (both) copy_packet(d + kBT, fv + kBT);
            if (fi + 1 < ncols) {
                copy_packet(d + 2 * kBT, fv + ld);
                if (both) copy_packet(d + 3 * kBT, fv + ld + kBT);
            }
        }
        copy_commit();
        fi += kUpCols;
        fv += kUpCols * ld;
        if (fi >= ncols) {                                    // the next pair
            fi = 0;
            fp += 2 * kBT;
            fv = vp + fp;
        }
        fo = fo == (kUpStages - 1) * kStage ? 0 : fo + kStage;
    };
#pragma unroll
    for (int k = 0; k < kUpStages - 1; ++k) fetch();
    PT nx[2];
    auto next = [&](int p) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (p + k * kBT < left) nx[k] = wp[p + k * kBT];
    };
    next(0);
    int uo = 0;
    for (int p = 0; p < pairs * 2 * kBT; p += 2 * kBT) {
        double2 acc[2][E];
#pragma unroll
        for (int k = 0; k < 2; ++k) P::get(nx[k], acc[k]);
        next(p + 2 * kBT);
        const double2* f = cs + rp;
        auto column = [&](const PT* d) {
            double2 y[2][E];
#pragma unroll
            for (int k = 0; k < 2; ++k) P::get(d[k * kBT], y[k]);
#pragma unroll
            for (int e = 0; e < E; ++e, f += PR) {
                const double2 c = *f;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    acc[k][e].x = fma(-c.x, y[k][e].x, acc[k][e].x);
                    acc[k][e].y = fma(-c.x, y[k][e].y, acc[k][e].y);
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    acc[k][e].x = fma(c.y, y[k][e].y, acc[k][e].x);
                    acc[k][e].y = fma(-c.y, y[k][e].x, acc[k][e].y);
                }
            }
        };
        for (int i = 0; i < ncols; i += kUpCols) {
            fetch();
            copy_wait<kUpStages - 1>();
            column(ring + uo);
            if (i + 1 < ncols) column(ring + uo + 2 * kBT);
            uo = uo == (kUpStages - 1) * kStage ? 0 : uo + kStage;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (p + k * kBT < left) {
                const PT o = P::put(acc[k]);
                wp[p + k * kBT] = o;
                double2 y[E];
                P::get(o, y);                                 // the norm of what is kept
#pragma unroll
                for (int e = 0; e < E; ++e) n2[e] += y[e].x * y[e].x + y[e].y * y[e].y;
            }
    }
    copy_wait<0>();
#pragma unroll
    for (int e = 0; e < E; ++e) {
        double s = n2[e];
#pragma unroll
        for (int o = PR; o < 32; o <<= 1) s += __shfl_xor_sync(kAll, s, o);
        if (lane < PR) rn[wid * NB + rp * E + e] = s;
    }
    __syncthreads();
    if (threadIdx.x < NB) {
        double s = 0.0;
        for (int k = 0; k < kBW; ++k) s += rn[k * NB + threadIdx.x];
        a.npart[(int64_t)blockIdx.x * NB + threadIdx.x] = s;
    }
}

template <typename VT, int NB>
__global__ void __launch_bounds__(kBT, 1) k_block_step(BlockStepArgs<VT> a) {
    using P = Pack<VT, NB>;
    using PT = typename P::T;
    constexpr int E = P::E, PR = NB / E;
    extern __shared__ double2 sm[];                   // a ring, the projections' sums; ring and coefficients
    double2* cs = sm + kUpStages * kUpCols * 2 * kBT * sizeof(PT) / sizeof(double2);
    __shared__ double rn[kBW * NB];
    __shared__ double before[NB], after[NB], alpha[NB];
    __shared__ int again[NB];
    if (*(volatile int*)a.err) return;                // an earlier launch of the solve gave up
    const int64_t r0 = (int64_t)blockIdx.x * a.rows;
    const int nr = (int)min((int64_t)a.rows, a.N - r0);
    const int nc = a.j + 1;
    VT* w = a.V + (int64_t)nc * a.N * NB;
    unsigned target = 0;
    for (int pass = 0; pass < 2; ++pass) {
        step_proj<VT, NB>(a, nc, pass == 0, r0, nr, w, sm, rn);
        if (!grid_barrier(a.bar, target, a.err)) return;
        step_reduce(a, (nc + (pass == 0 ? 1 : 0)) * NB);
        if (!grid_barrier(a.bar, target, a.err)) return;
        for (int e = threadIdx.x; e < nc * NB; e += kBT) {
            const int i = e / NB, r = e % NB;
            double2 c = __ldcg(a.coef + e);
            if (i == a.j) {
                if (pass == 0) alpha[r] = c.x;
                else if (again[r]) alpha[r] += c.x;
            }
            if (pass == 1 && !again[r]) c = make_double2(0.0, 0.0);
            cs[(i * E + r % E) * PR + r / E] = c;
        }
        if (pass == 0 && threadIdx.x < NB) before[threadIdx.x] = __ldcg(a.coef + nc * NB + threadIdx.x).x;
        __syncthreads();
        step_update<VT, NB>(a, nc, r0, nr, w, sm, cs, rn);
        if (!grid_barrier(a.bar, target, a.err)) return;
        // |w_r|^2 over the blocks: kBT / NB runs of blocks, then the runs
        {
            const int r = threadIdx.x % NB;
            double s = 0.0;
            for (int b = threadIdx.x / NB; b < (int)gridDim.x; b += kBT / NB) s += __ldcg(a.npart + (int64_t)b * NB + r);
            double* runs = reinterpret_cast<double*>(sm);
            runs[threadIdx.x] = s;
            __syncthreads();
            if (threadIdx.x < NB) {
                s = 0.0;
                for (int k = 0; k < kBT / NB; ++k) s += runs[k * NB + r];
                after[r] = s;
                if (pass == 0) again[r] = s < a.keep * before[r] ? 1 : 0;
            }
            __syncthreads();
        }
        if (pass == 0) {
            int any = 0;
            for (int r = 0; r < NB; ++r) any |= again[r];
            if (!any) break;                          // the same in every block
        }
    }
    double sc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const double b = sqrt(max(after[threadIdx.x % PR * E + e], 0.0));
        sc[e] = b > 0.0 ? 1.0 / b : 0.0;
    }
    PT* wp = reinterpret_cast<PT*>(w) + r0 * PR;
#pragma unroll 4
    for (int p = threadIdx.x; p < nr * PR; p += kBT) {
        double2 y[E];
        P::get(wp[p], y);
#pragma unroll
        for (int e = 0; e < E; ++e) y[e] = make_double2(y[e].x * sc[e], y[e].y * sc[e]);
        wp[p] = P::put(y);
    }
    if (blockIdx.x == 0 && threadIdx.x < NB) {
        a.alpha[threadIdx.x * a.m + a.j] = alpha[threadIdx.x];
        a.beta[threadIdx.x * a.m + a.j] = sqrt(max(after[threadIdx.x], 0.0));
    }
    barrier_exit(a.bar);
}

template <typename VT> size_t step_smem(int nb, int m) {
    const size_t pt = std::is_same<VT, float2>::value && nb == 1 ? 8 : 16;    // a packet
    return std::max({(size_t)kStages * (kCG + 1) * kBT * pt, (size_t)kBW * kCG * nb * sizeof(double2),
                     (size_t)kUpStages * kUpCols * 2 * kBT * pt + (size_t)m * nb * sizeof(double2)});
}

template <typename VT> const void* step_kernel(int nb) {
    switch (nb) {
        case 1: return reinterpret_cast<const void*>(k_block_step<VT, 1>);
        case 2: return reinterpret_cast<const void*>(k_block_step<VT, 2>);
        case 4: return reinterpret_cast<const void*>(k_block_step<VT, 4>);
        case 8: return reinterpret_cast<const void*>(k_block_step<VT, 8>);
        case 16: return reinterpret_cast<const void*>(k_block_step<VT, 16>);
        case 32: return reinterpret_cast<const void*>(k_block_step<VT, 32>);
        default: return nullptr;
    }
}

}  // namespace

template <typename VT>
bool block_step_plan(int64_t N, int nb, int m, BlockStepArgs<VT>& a, int& grid) {
    const void* k = step_kernel<VT>(nb);
    if (N < 1 || !k || m < 1 || m > kMaxCols) return false;
    int dev = 0, sms = 0, coop = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    // process-wide attribute: always the largest size, so concurrent callers never lower it
    MOMED_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)step_smem<VT>(nb, kMaxCols)));
    MOMED_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kBT, step_smem<VT>(nb, m)));
    if (!coop || per < 1 || sms < 1) return false;
    const int64_t rows = std::max<int64_t>((N + sms - 1) / sms, std::min(kBT / nb, 32));   // a value per thread or more
    if (rows * nb >= (int64_t)1 << 30) return false;
    a.N = N;
    a.rows = (int)rows;
    grid = (int)((N + rows - 1) / rows);
    return true;
}

template <typename VT>
bool launch_block_step(const BlockStepArgs<VT>& a, int nb, int grid, cudaStream_t st) {
    void* args[] = {const_cast<BlockStepArgs<VT>*>(&a)};
    return launch_cooperative(step_kernel<VT>(nb), grid, kBT, args, step_smem<VT>(nb, a.m), st);
}

template bool block_step_plan<double2>(int64_t, int, int, BlockStepArgs<double2>&, int&);
template bool block_step_plan<float2>(int64_t, int, int, BlockStepArgs<float2>&, int&);
template bool launch_block_step<double2>(const BlockStepArgs<double2>&, int, int, cudaStream_t);
template bool launch_block_step<float2>(const BlockStepArgs<float2>&, int, int, cudaStream_t);

}  // namespace momed
