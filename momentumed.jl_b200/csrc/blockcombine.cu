// Recombinations of block vectors: the restart of the lockstep solver, its Ritz vectors, and the
// refinement's X' = [X Q] Y.
//
// A thread owns one 16-byte packet of a row (two packets in the complex form) and keeps the sums of up
// to 16 outputs in registers, so V is read once for all of them; the coefficients, packed by the host in
// the arithmetic's type and padded to whole tiles, come from L1 as one load per output.  The packets
// themselves run ahead through a ring in shared memory, beyond what the registers of a loop could hold.
//
// What bounds it: HBM, and L1 for the coefficients (a 12-output source costs 12 loads beside one packet).
// Measured on 173.6k states x 32 right-hand sides (44 MB a c64 column): restart of 30 columns to 12, c64,
// 1.23 -> 0.54 ms (1.9 GB, floor 0.29; from registers alone, four loads ahead, 0.75); Ritz vectors of 8
// FP64 blocks 1.76 ms and [X Q] Y of 8 FP64 and 25 FP32 blocks 1.21 ms -> 0.69 ms on average, where each
// coefficient was converted to FP32 by every thread and the FP64 form read its sources once per output.
#include <algorithm>
#include <type_traits>

#include "blockcombine.cuh"
#include "packets.cuh"

namespace momed {

namespace {

constexpr int kT = 256;
constexpr int kStages = 4, kRun = 4;   // ring of k_block_combine: runs of 4 sources, 64 KB of 16-byte packets
constexpr int kStagesC = 8;            // ring of k_block_combine_c: two values of a source, 64 KB
constexpr size_t kRing = (size_t)kStages * kRun * kT * 16;
static_assert(kRing == (size_t)kStagesC * 2 * kT * 16, "both rings");

int combine_sms() {
    static const int s = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 148;
    }();
    return s;
}

// E adjacent values of VT
template <typename VT, int E> struct Vals;
template <> struct Vals<float2, 2> { using T = float4; };
template <> struct Vals<float2, 1> { using T = float2; };
template <> struct Vals<double2, 1> { using T = double2; };
template <typename R, int E> struct Coef;
template <> struct Coef<float, 2> { using T = float2; };
template <> struct Coef<float, 1> { using T = float; };
template <> struct Coef<double, 2> { using T = double2; };
template <> struct Coef<double, 1> { using T = double; };

template <typename PT, typename R, int E> __device__ __forceinline__ void split(const PT& p, R* x, R* y) {
    x[0] = (R)p.x;
    y[0] = (R)p.y;
    if constexpr (E == 2) {
        x[1] = (R)p.z;
        y[1] = (R)p.w;
    }
}

// U: [m][tiles OC][nb]; total: packets of a column; grid.y: tiles of OC outputs
template <typename VIN, typename VOUT, typename R, int E, int OC>
__global__ void __launch_bounds__(kT, OC * E * sizeof(R) > 64 ? 2 : 3)
k_block_combine(const VIN* __restrict__ V, int64_t total, int nb, int m, const R* __restrict__ U, int nout,
                VOUT* __restrict__ out, int copy_col) {
    using PT = typename Vals<VIN, E>::T;
    using CT = typename Coef<R, E>::T;
    const int c0 = blockIdx.y * OC, pr = nb / E;
    const int64_t cs = (int64_t)gridDim.y * OC * pr;                // coefficients of one source, in CT
    const PT* Vp = reinterpret_cast<const PT*>(V);
    extern __shared__ double2 sm[];
    PT* ring = reinterpret_cast<PT*>(sm) + threadIdx.x;
    int64_t fe = (int64_t)blockIdx.x * kT + threadIdx.x;            // the next copy: packet, source, stage
    int fa = 0, fo = 0, uo = 0;
    auto fetch = [&] {
        if (fe < total) {
            const PT* v = Vp + fa * total + fe;
#pragma unroll
            for (int k = 0; k < kRun; ++k, v += total)
                if (fa + k < m) copy_packet(ring + fo + k * kT, v);
        }
        copy_commit();
        fa += kRun;
        if (fa >= m) {
            fa = 0;
            fe += (int64_t)gridDim.x * kT;
        }
        fo = fo == (kStages - 1) * kRun * kT ? 0 : fo + kRun * kT;
    };
#pragma unroll
    for (int k = 0; k < kStages - 1; ++k) fetch();
    for (int64_t e = (int64_t)blockIdx.x * kT + threadIdx.x; e < total; e += (int64_t)gridDim.x * kT) {
        const CT* up = reinterpret_cast<const CT*>(U) + (int64_t)c0 * pr + (e & (pr - 1));
        R ax[OC][E], ay[OC][E];
#pragma unroll
        for (int c = 0; c < OC; ++c)
#pragma unroll
            for (int q = 0; q < E; ++q) ax[c][q] = ay[c][q] = 0;
        auto add = [&](const PT& v) {
            R x[E], y[E];
            split<PT, R, E>(v, x, y);
#pragma unroll
            for (int c = 0; c < OC; ++c) {
                const CT u = __ldg(up + c * pr);
                R uq[E];
                if constexpr (E == 2) {
                    uq[0] = u.x;
                    uq[1] = u.y;
                } else {
                    uq[0] = u;
                }
#pragma unroll
                for (int q = 0; q < E; ++q) {
                    ax[c][q] += uq[q] * x[q];
                    ay[c][q] += uq[q] * y[q];
                }
            }
            up += cs;
        };
        for (int a = 0; a < m; a += kRun) {
            fetch();
            copy_wait<kStages - 1>();
            const PT* d = ring + uo;
            const int n = min(kRun, m - a);
#pragma unroll 1
            for (int k = 0; k < n; ++k) add(d[k * kT]);
            uo = uo == (kStages - 1) * kRun * kT ? 0 : uo + kRun * kT;
        }
#pragma unroll
        for (int c = 0; c < OC; ++c)
            if (c0 + c < nout) {
                VOUT* o = out + ((int64_t)(c0 + c) * total + e) * E;
#pragma unroll
                for (int q = 0; q < E; ++q) {
                    o[q].x = ax[c][q];
                    o[q].y = ay[c][q];
                }
            }
        if (copy_col >= 0 && blockIdx.y == 0) {
            R x[E], y[E];
            split<PT, R, E>(Vp[(int64_t)copy_col * total + e], x, y);
            VOUT* o = out + ((int64_t)nout * total + e) * E;
#pragma unroll
            for (int q = 0; q < E; ++q) {
                o[q].x = x[q];
                o[q].y = y[q];
            }
        }
    }
}

// Y64: [kx + kz][tiles OC][nb], Y32: [p][tiles OC][nb]; a thread owns values e and e + half (half a
// multiple of nb, so both are of one right-hand side)
template <int OC>
__global__ void __launch_bounds__(kT, 2)
k_block_combine_c(const double2* __restrict__ X, int kx, const double2* __restrict__ Z, int kz,
                  const float2* __restrict__ Q, int p, int64_t total, int64_t half, int nb,
                  const double2* __restrict__ Y64, const float2* __restrict__ Y32, int nout, double2* __restrict__ out) {
    const int c0 = blockIdx.y * OC;
    const int64_t cs = (int64_t)gridDim.y * OC * nb;
    extern __shared__ double2 sm[];
    double2* ring = sm + threadIdx.x;
    const int d = p + kx + kz;
    int64_t fe = (int64_t)blockIdx.x * kT + threadIdx.x;            // the next copy: value, source (Q, X, Z), stage
    int fa = 0, fo = 0, uo = 0;
    auto fetch = [&] {
        if (fe < half) {
            const int64_t f1 = fe + half < total ? fe + half : fe;
            if (fa < p) {
                const float2* q = Q + fa * total;
                copy_packet(reinterpret_cast<float2*>(ring + fo), q + fe);
                copy_packet(reinterpret_cast<float2*>(ring + fo + kT), q + f1);
            } else {
                const double2* x = fa < p + kx ? X + (fa - p) * total : Z + (fa - p - kx) * total;
                copy_packet(ring + fo, x + fe);
                copy_packet(ring + fo + kT, x + f1);
            }
        }
        copy_commit();
        if (++fa == d) {
            fa = 0;
            fe += (int64_t)gridDim.x * kT;
        }
        fo = fo == (kStagesC - 1) * 2 * kT ? 0 : fo + 2 * kT;
    };
    auto arrive = [&] {                                             // the stage of the next source
        fetch();
        copy_wait<kStagesC - 1>();
        const double2* at = ring + uo;
        uo = uo == (kStagesC - 1) * 2 * kT ? 0 : uo + 2 * kT;
        return at;
    };
#pragma unroll
    for (int k = 0; k < kStagesC - 1; ++k) fetch();
    for (int64_t e0 = (int64_t)blockIdx.x * kT + threadIdx.x; e0 < half; e0 += (int64_t)gridDim.x * kT) {
        const int64_t e1 = e0 + half;
        const bool two = e1 < total;
        const int64_t co = (int64_t)c0 * nb + (e0 & (nb - 1));
        double ax[2][OC], ay[2][OC];
        {
            float fx[2][OC], fy[2][OC];
#pragma unroll
            for (int c = 0; c < OC; ++c) fx[0][c] = fy[0][c] = fx[1][c] = fy[1][c] = 0.f;
            const float2* yp = Y32 + co;
#pragma unroll 1
            for (int a = 0; a < p; ++a, yp += cs) {
                const double2* at = arrive();
                const float2 v0 = *reinterpret_cast<const float2*>(at), v1 = *reinterpret_cast<const float2*>(at + kT);
#pragma unroll
                for (int c = 0; c < OC; ++c) {
                    const float2 y = __ldg(yp + c * nb);
                    fx[0][c] += y.x * v0.x - y.y * v0.y;
                    fy[0][c] += y.x * v0.y + y.y * v0.x;
                    fx[1][c] += y.x * v1.x - y.y * v1.y;
                    fy[1][c] += y.x * v1.y + y.y * v1.x;
                }
            }
#pragma unroll
            for (int c = 0; c < OC; ++c)
#pragma unroll
                for (int k = 0; k < 2; ++k) { ax[k][c] = (double)fx[k][c]; ay[k][c] = (double)fy[k][c]; }
        }
        const double2* yp = Y64 + co;
#pragma unroll 1
        for (int a = 0; a < kx + kz; ++a, yp += cs) {
            const double2* at = arrive();
            const double2 v0 = at[0], v1 = at[kT];
#pragma unroll
            for (int c = 0; c < OC; ++c) {
                const double2 y = __ldg(yp + c * nb);
                ax[0][c] = fma(-y.y, v0.y, fma(y.x, v0.x, ax[0][c]));
                ay[0][c] = fma(y.y, v0.x, fma(y.x, v0.y, ay[0][c]));
                ax[1][c] = fma(-y.y, v1.y, fma(y.x, v1.x, ax[1][c]));
                ay[1][c] = fma(y.y, v1.x, fma(y.x, v1.y, ay[1][c]));
            }
        }
#pragma unroll
        for (int c = 0; c < OC; ++c)
            if (c0 + c < nout) {
                out[(c0 + c) * total + e0] = make_double2(ax[0][c], ay[0][c]);
                if (two) out[(c0 + c) * total + e1] = make_double2(ax[1][c], ay[1][c]);
            }
    }
}

// Tiles of the outputs: as few as hold at most most each, evenly sized, rounded up to a multiple of step
struct Tiles {
    int count, size;
    Tiles(int nout, int most, int step) {
        count = (nout + most - 1) / most;
        size = (nout + count - 1) / count;
        size = (size + step - 1) / step * step;
    }
};

template <typename VIN, typename VOUT, typename R, int E>
void combine_launch(const VIN* V, int64_t total, int nb, int m, const R* U, int nout, VOUT* out, int copy_col, Tiles t,
                    cudaStream_t st) {
    const dim3 grid((unsigned)std::min<int64_t>((total + kT - 1) / kT, (int64_t)combine_sms() * 16), (unsigned)t.count);
    auto go = [&](auto k) {
        MOMED_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRing));
        k<<<grid, kT, kRing, st>>>(V, total, nb, m, U, nout, out, copy_col);
    };
    switch (t.size) {
        case 4: go(k_block_combine<VIN, VOUT, R, E, 4>); break;
        case 8: go(k_block_combine<VIN, VOUT, R, E, 8>); break;
        case 12:
            if constexpr (!(std::is_same<R, double>::value && E == 2))
                go(k_block_combine<VIN, VOUT, R, E, 12>);
            break;
        default:
            if constexpr (!(std::is_same<R, double>::value && E == 2))
                go(k_block_combine<VIN, VOUT, R, E, 16>);
            break;
    }
    MOMED_CUDA_TRY(cudaGetLastError());
}

}  // namespace

template <typename VIN, typename VOUT>
void block_combine(const VIN* V, int64_t N, int nb, int m, const std::vector<double>& U, int nout, VOUT* out,
                   int copy_col, DevBuf<double>& buf, cudaStream_t st) {
    constexpr bool f32 = std::is_same<VIN, float2>::value && std::is_same<VOUT, float2>::value;
    using R = typename std::conditional<f32, float, double>::type;
    const bool wide = std::is_same<VIN, float2>::value && nb % 2 == 0;
    // 16 outputs keep 64 registers of sums (two FP32 or one FP64 value each), 8 the same with two FP64
    const Tiles t(nout, wide && !f32 ? 8 : 16, 4);
    const int op = t.count * t.size;
    std::vector<R> u((size_t)m * op * nb, R(0));
    for (int i = 0; i < nout; ++i)
        for (int a = 0; a < m; ++a)
            for (int r = 0; r < nb; ++r) u[((size_t)a * op + i) * nb + r] = (R)U[((size_t)i * m + a) * nb + r];
    buf.resize(u.size() * sizeof(R) / sizeof(double) + 1);
    R* ud = reinterpret_cast<R*>(buf.p);
    MOMED_CUDA_TRY(cudaMemcpyAsync(ud, u.data(), u.size() * sizeof(R), cudaMemcpyHostToDevice, st));
    if constexpr (std::is_same<VIN, float2>::value) {
        if (wide) {
            combine_launch<VIN, VOUT, R, 2>(V, N * nb / 2, nb, m, ud, nout, out, copy_col, t, st);
            return;
        }
    }
    combine_launch<VIN, VOUT, R, 1>(V, N * nb, nb, m, ud, nout, out, copy_col, t, st);
}

void block_combine_c(const double2* X, int kx, const double2* Z, int kz, const float2* Q, int p, int64_t N, int nb,
                     const std::vector<double2>& Y, int nout, double2* out, DevBuf<double2>& buf, cudaStream_t st) {
    const int d = kx + kz + p;
    const Tiles t(nout, 8, 2);
    const int op = t.count * t.size;
    // one upload: the FP64 sources' coefficients, then the FP32 source's in FP32
    const size_t n64 = (size_t)(kx + kz) * op * nb, n32 = (size_t)p * op * nb;
    std::vector<double2> y(n64 + (n32 + 1) / 2, make_double2(0.0, 0.0));
    float2* y32 = reinterpret_cast<float2*>(y.data() + n64);
    for (int i = 0; i < nout; ++i)
        for (int a = 0; a < d; ++a)
            for (int r = 0; r < nb; ++r) {
                const double2 v = Y[((size_t)i * d + a) * nb + r];
                if (a < kx + kz) y[((size_t)a * op + i) * nb + r] = v;
                else y32[((size_t)(a - kx - kz) * op + i) * nb + r] = make_float2((float)v.x, (float)v.y);
            }
    buf.resize(std::max<size_t>(y.size(), 1));
    MOMED_CUDA_TRY(cudaMemcpyAsync(buf.p, y.data(), y.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
    const int64_t total = N * nb, half = (N + 1) / 2 * nb;
    const dim3 grid((unsigned)std::min<int64_t>((half + kT - 1) / kT, (int64_t)combine_sms() * 16), (unsigned)t.count);
    const double2* y64 = buf.p;
    const float2* yq = reinterpret_cast<const float2*>(buf.p + n64);
    auto go = [&](auto k) {
        MOMED_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRing));
        k<<<grid, kT, kRing, st>>>(X, kx, Z, kz, Q, p, total, half, nb, y64, yq, nout, out);
    };
    switch (t.size) {
        case 2: go(k_block_combine_c<2>); break;
        case 4: go(k_block_combine_c<4>); break;
        case 6: go(k_block_combine_c<6>); break;
        default: go(k_block_combine_c<8>); break;
    }
    MOMED_CUDA_TRY(cudaGetLastError());
}

template void block_combine<float2, float2>(const float2*, int64_t, int, int, const std::vector<double>&, int, float2*, int, DevBuf<double>&, cudaStream_t);
template void block_combine<float2, double2>(const float2*, int64_t, int, int, const std::vector<double>&, int, double2*, int, DevBuf<double>&, cudaStream_t);
template void block_combine<double2, double2>(const double2*, int64_t, int, int, const std::vector<double>&, int, double2*, int, DevBuf<double>&, cudaStream_t);

}  // namespace momed
