// Lanczos steps of the single-vector solvers as one cooperative kernel.
//
// A step of lanczos.cu (and of batch.cu with one right-hand side) is a map and nine vector kernels (projection, reduction, update, the test
// for a second Gram-Schmidt pass, that pass, the norm, the scaling), most of them a few
// microseconds: on sectors of a few hundred to some ten thousand states a solve spends its time on
// launches.  Here a block owns a contiguous range of rows for the whole launch and keeps its part of
// w in shared memory; the blocks meet at two grid barriers per step (after the projections, after
// the norm) and every block sums the blocks' partial results itself, in the same fixed order, so
// all of them take the same decisions:
//
//   w = s H x          the rows of the block (x: the last vector before its scaling, s = 1 / beta)
//   c_i = V_i^H w      per-block partials                      | barrier
//   w -= sum c_i V_i   |w|^2 per block, w written for the maps | barrier
//   (both once more when less than a tenth of |w|^2 is left)
//   V_{j+1} = w / beta the block's own rows, read by itself alone until the launch ends
//
// With the map inside (hit records or CSR) one launch runs all steps of a restart cycle.  Beside the
// pair-factorised map, whose first stage wants other blocks and registers, a launch runs one step's
// orthogonalisation (MAP_NONE).
//
// What bounds it: two barriers (about 1.2 us each over 148 blocks) and the map's gathers on small
// sectors, the two reads of V on large ones.  One FP64 solve of 4 pairs on the B200, separate kernels
// / this: 200 states 2.97 / 1.18 ms, 5.5k 8.05 / 3.58, 30.6k 13.1 / 7.1, 104k (hit records) 26.1 /
// 19.2, 276k (beside the pair map) 41.8 / 34.3, 1.0M 266 / 250: it wins at every size, so the
// separate kernels stay for what it does not do (per-launch timing, candidate and slot-mode maps,
// FP32 steps of lanczos.cu, more rows than the blocks' shared memory holds: 1.7M states in FP64).
#include <algorithm>
#include <type_traits>

#include "cycle.cuh"

namespace momed {

namespace {

constexpr int kCT = 1024;              // threads per block, one block per SM
constexpr int kCW = kCT / 32;
constexpr unsigned kAll = 0xffffffffu;
constexpr int kMaxChunks = 8;          // row chunks of a block's projections
constexpr size_t kMaxSmem = 200 * 1024;

__device__ __forceinline__ double wred(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
    return v;
}
__device__ __forceinline__ uint2 ld_rec(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ int32_t ld_rec(const int32_t* p) {
    int32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 ld_rec(const double2* p) {
    double2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// w[r] = s * (H x)[r0 + r], a warp per row as k_matvec_hc and k_spmv do it
template <int MAP>
__device__ __forceinline__ void cycle_map(const CycleArgs<double2>& a, const double2* x, double s, int64_t r0, int nr, double2* w) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int r = wid; r < nr; r += kCW) {
        const int64_t row = r0 + r;
        const int64_t b = __ldg(a.row_ptr + row), e = __ldg(a.row_ptr + row + 1);
        double ar = 0.0, ai = 0.0;
        int64_t p = b + lane;
        auto one = [&](double2 v, double2 xv) {
            ar += v.x * xv.x - v.y * xv.y;
            ai += v.x * xv.y + v.y * xv.x;
        };
        if constexpr (MAP == CYCLE_HITS) {
            auto val = [&](uint32_t tw) {
                double2 v = __ldg(a.amp + (tw & 0x7fffffffu));
                if (tw >> 31) { v.x = -v.x; v.y = -v.y; }
                return v;
            };
            for (; p + 96 < e; p += 128) {
                uint2 h[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) h[q] = ld_rec(a.hit + p + 32 * q);
#pragma unroll
                for (int q = 0; q < 4; ++q) one(val(h[q].y), x[h[q].x]);
            }
            for (; p < e; p += 32) {
                const uint2 h = ld_rec(a.hit + p);
                one(val(h.y), x[h.x]);
            }
        } else {
            for (; p + 96 < e; p += 128) {
                int32_t c[4];
                double2 v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    c[q] = ld_rec(a.col + p + 32 * q);
                    v[q] = ld_rec(a.val + p + 32 * q);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) one(v[q], x[c[q]]);
            }
            for (; p < e; p += 32) one(ld_rec(a.val + p), x[ld_rec(a.col + p)]);
        }
        ar = wred(ar);
        ai = wred(ai);
        if (lane == 0) {
            if constexpr (MAP == CYCLE_HITS) {
                double2 d = __ldg(a.dg + 2 * row);
                if (a.has_b) {
                    const double2 db = __ldg(a.dg + 2 * row + 1);
                    d.x += a.u * db.x;
                    d.y += a.u * db.y;
                }
                const double2 xd = x[row];
                ar += d.x * xd.x - d.y * xd.y;
                ai += d.x * xd.y + d.y * xd.x;
            }
            w[r] = make_double2(s * ar, s * ai);
        }
    }
}

// part[c][block] = the block's share of V_c^H w for c < ncols (and |w|^2 as c = ncols when norm)
template <typename VT>
__device__ __forceinline__ void cycle_proj(const CycleArgs<VT>& a, int ncols, bool norm, int64_t r0, int nr, const VT* w,
                                           double2* slot) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ch = a.chunks, len = (nr + ch - 1) / ch, total = (ncols + (norm ? 1 : 0)) * ch;
    for (int t = wid; t < total; t += kCW) {
        const int c = t / ch, q = t - c * ch;
        const int b = q * len, e = min(nr, b + len);
        double ax = 0.0, ay = 0.0;
        if (c < ncols) {
            const VT* v = a.V + (int64_t)c * a.N + r0;
#pragma unroll 4
            for (int r = b + lane; r < e; r += 32) {
                const double2 vv = to_d2(v[r]), ww = to_d2(w[r]);
                ax += vv.x * ww.x + vv.y * ww.y;
                ay += vv.x * ww.y - vv.y * ww.x;
            }
        } else {
            for (int r = b + lane; r < e; r += 32) {
                const double2 ww = to_d2(w[r]);
                ax += ww.x * ww.x + ww.y * ww.y;
            }
        }
        ax = wred(ax);
        ay = wred(ay);
        if (lane == 0) slot[t] = make_double2(ax, ay);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < total / ch; c += kCT) {
        double2 s = make_double2(0.0, 0.0);
        for (int q = 0; q < ch; ++q) { s.x += slot[c * ch + q].x; s.y += slot[c * ch + q].y; }
        a.part[(int64_t)c * gridDim.x + blockIdx.x] = s;
    }
}

// coef[c] = sum over the blocks, the same order in every block
template <typename VT>
__device__ __forceinline__ void cycle_reduce(const CycleArgs<VT>& a, int count, double2* coef) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int c = wid; c < count; c += kCW) {
        const double2* p = a.part + (int64_t)c * gridDim.x;
        double sx = 0.0, sy = 0.0;
        for (int g = lane; g < (int)gridDim.x; g += 32) {
            const double2 v = __ldcg(p + g);
            sx += v.x;
            sy += v.y;
        }
        sx = wred(sx);
        sy = wred(sy);
        if (lane == 0) coef[c] = make_double2(sx, sy);
    }
    __syncthreads();
}

// w -= sum_i coef[i] V_i on the block's rows, S lanes per row; the block's |w|^2 to npart, w to xn
template <typename VT>
__device__ __forceinline__ void cycle_update(const CycleArgs<VT>& a, int ncols, int64_t r0, int nr, VT* w,
                                             const double2* coef, VT* xn, double* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int S = a.split, rl = 32 / S, s = lane / rl;
    double n2 = 0.0;
    for (int rb = wid * rl; rb < nr; rb += kCW * rl) {        // warp-uniform
        const int r = rb + lane % rl;
        const bool in = r < nr;
        double ax = 0.0, ay = 0.0;
        if (in) {
            const VT* v = a.V + r0 + r;
#pragma unroll 4
            for (int i = s; i < ncols; i += S) {
                const double2 c = coef[i], vv = to_d2(v[(int64_t)i * a.N]);
                ax += c.x * vv.x - c.y * vv.y;
                ay += c.x * vv.y + c.y * vv.x;
            }
        }
        for (int o = rl; o < 32; o <<= 1) {
            ax += __shfl_xor_sync(kAll, ax, o);
            ay += __shfl_xor_sync(kAll, ay, o);
        }
        if (in && s == 0) {
            const double2 wv = to_d2(w[r]);
            const VT v = from_d2<VT>(make_double2(wv.x - ax, wv.y - ay));
            w[r] = v;
            if (xn) xn[r0 + r] = v;
            const double2 back = to_d2(v);           // the norm of what is kept
            n2 += back.x * back.x + back.y * back.y;
        }
    }
    n2 = wred(n2);
    if (lane == 0) red[wid] = n2;
    __syncthreads();
    if (wid == 0) {
        const double v = wred(red[lane]);
        if (lane == 0) a.npart[blockIdx.x] = v;
    }
}

// |w|^2 over all blocks (every thread)
template <typename VT>
__device__ __forceinline__ double cycle_norm(const CycleArgs<VT>& a, double* red) {
    const int lane = threadIdx.x & 31;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = 0.0;
        for (int g = lane; g < (int)gridDim.x; g += 32) v += __ldcg(a.npart + g);
        v = wred(v);
        if (lane == 0) red[0] = v;
    }
    __syncthreads();
    const double v = red[0];
    __syncthreads();
    return v;
}

template <typename VT, int MAP>
__global__ void __launch_bounds__(kCT, 1) k_lanczos_cycle(CycleArgs<VT> a) {
    extern __shared__ double2 sm[];
    double2* coef = sm;                              // [kMaxCols + 1]
    double2* slot = coef + kMaxCols + 1;             // [(kMaxCols + 1) * chunks]
    VT* w = reinterpret_cast<VT*>(slot + (kMaxCols + 1) * a.chunks);   // [rows]
    __shared__ double red[kCW];
    if (*(volatile int*)a.err) return;               // an earlier launch of the solve gave up
    const int64_t r0 = (int64_t)blockIdx.x * a.rows;
    const int nr = (int)max((int64_t)0, min((int64_t)a.rows, a.N - r0));
    unsigned target = 0;
    double s = 1.0;
    const VT* x = a.V + (int64_t)a.j0 * a.N;
    for (int j = a.j0; j < a.j1; ++j) {
        const int nc = j + 1;
        VT* vn = a.V + (int64_t)nc * a.N;
        VT* xn = nullptr;
        if constexpr (MAP != CYCLE_NONE) xn = a.xbuf + (int64_t)(j & 1) * a.N;
        if constexpr (MAP == CYCLE_NONE) {
            for (int r = threadIdx.x; r < nr; r += kCT) w[r] = vn[r0 + r];
        } else {
            cycle_map<MAP>(a, x, s, r0, nr, w);
        }
        __syncthreads();
        cycle_proj(a, nc, true, r0, nr, w, slot);
        if (!grid_barrier(a.bar, target, a.err)) return;
        cycle_reduce(a, nc + 1, coef);
        const double before = coef[nc].x;
        double alpha = coef[j].x;
        cycle_update(a, nc, r0, nr, w, coef, xn, red);
        if (!grid_barrier(a.bar, target, a.err)) return;
        double after = cycle_norm(a, red);
        if (after < a.keep * before) {
            cycle_proj(a, nc, false, r0, nr, w, slot);
            if (!grid_barrier(a.bar, target, a.err)) return;
            cycle_reduce(a, nc, coef);
            alpha += coef[j].x;
            cycle_update(a, nc, r0, nr, w, coef, xn, red);
            if (!grid_barrier(a.bar, target, a.err)) return;
            after = cycle_norm(a, red);
        }
        const double b = sqrt(max(after, 0.0));
        s = b > 0.0 ? 1.0 / b : 0.0;
        for (int r = threadIdx.x; r < nr; r += kCT) {
            const double2 v = to_d2(w[r]);
            vn[r0 + r] = from_d2<VT>(make_double2(v.x * s, v.y * s));
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.alpha[j] = alpha;
            a.beta[j] = b;
        }
        x = xn;
        __syncthreads();                             // w is written again by the next step
    }
    barrier_exit(a.bar);
}

int cycle_sms() {
    static const int s = [] {
        int dev = 0, v = 0, coop = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        return coop ? v : 0;
    }();
    return s;
}

size_t cycle_smem(int rows, int chunks, size_t elem) {
    return (kMaxCols + 1) * (size_t)(1 + chunks) * sizeof(double2) + (size_t)rows * elem;
}

}  // namespace

template <typename VT> static const void* cycle_kernel(int map) {
    if constexpr (std::is_same<VT, double2>::value) {
        if (map == CYCLE_HITS) return reinterpret_cast<const void*>(k_lanczos_cycle<double2, CYCLE_HITS>);
        if (map == CYCLE_CSR) return reinterpret_cast<const void*>(k_lanczos_cycle<double2, CYCLE_CSR>);
    }
    return reinterpret_cast<const void*>(k_lanczos_cycle<VT, CYCLE_NONE>);
}

// Small sectors take at least 32 rows a block (a barrier over few blocks is shorter).
template <typename VT>
bool cycle_plan(int64_t N, int map, CycleArgs<VT>& a, int& grid) {
    const int sms = cycle_sms();
    if (N < 1 || sms < 1) return false;
    const int64_t rows = std::max<int64_t>(32, (N + sms - 1) / sms);
    if (rows > (int64_t)(kMaxSmem / sizeof(VT))) return false;
    a.N = N;
    a.rows = (int)rows;
    a.chunks = (int)std::min<int64_t>(kMaxChunks, std::max<int64_t>(1, rows / 128));
    a.split = rows <= 512 ? 4 : rows <= 2048 ? 2 : 1;
    grid = (int)((N + rows - 1) / rows);
    const size_t smem = cycle_smem(a.rows, a.chunks, sizeof(VT));
    if (smem > kMaxSmem) return false;
    // process-wide attribute: always the largest size, so concurrent callers never lower it
    const void* k = cycle_kernel<VT>(map);
    int per = 0;
    MOMED_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
    MOMED_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kCT, smem));
    return per >= 1;
}

template <typename VT>
bool launch_cycle(CycleArgs<VT>& a, int map, int grid, cudaStream_t st) {
    void* args[] = {&a};
    return launch_cooperative(cycle_kernel<VT>(map), grid, kCT, args, cycle_smem(a.rows, a.chunks, sizeof(VT)), st);
}

template bool cycle_plan<double2>(int64_t, int, CycleArgs<double2>&, int&);
template bool cycle_plan<float2>(int64_t, int, CycleArgs<float2>&, int&);
template bool launch_cycle<double2>(CycleArgs<double2>&, int, int, cudaStream_t);
template bool launch_cycle<float2>(CycleArgs<float2>&, int, int, cudaStream_t);

}  // namespace momed
