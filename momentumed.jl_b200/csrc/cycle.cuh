// Cooperative kernels for Lanczos steps: a single-vector cycle (cycle.cu), a step of the lockstep block
// solver (blockstep.cu).
#pragma once
#include <cstdlib>

#include "vecops.cuh"

namespace momed {

#ifdef __CUDACC__
constexpr uint64_t kWaitNs = 2000000000ull;   // a barrier gives up after two seconds
__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// All blocks of the cooperative launch arrive; what they wrote before is visible after.  False (for
// every thread of the block) when the wait ran out: the kernel then returns and the host reads err.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned& target, int* err) {
    __shared__ int ok;
    __syncthreads();
    if (gridDim.x == 1) return true;
    if (threadIdx.x == 0) {
        target += gridDim.x;
        ok = 1;
        __threadfence();
        atomicAdd(bar, 1u);
        const uint64_t t0 = now_ns();
        while (ld_acquire(bar) < target) {
            if (now_ns() - t0 > kWaitNs) {
                atomicExch(err, 1);
                ok = 0;
                break;
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

// the last block out leaves the barrier as it found it
__device__ __forceinline__ void barrier_exit(unsigned* bar) {
    if (threadIdx.x == 0 && gridDim.x > 1 && atomicAdd(bar + 1, 1u) == gridDim.x - 1) {
        bar[0] = 0u;
        bar[1] = 0u;
        __threadfence();
    }
}
#endif

enum CycleMap : int { CYCLE_NONE = 0, CYCLE_HITS = 1, CYCLE_CSR = 2 };

// VT: the basis, double2 or float2 (FP32 vectors, FP64 sums; the map beside it only).
template <typename VT> struct CycleArgs {
    VT* V;                     // basis, column i at V + i N
    int64_t N;
    int j0, j1;                // steps [j0, j1); column j0 is normalised
    int rows, chunks, split;   // cycle_plan
    double2* part;             // [kMaxCols + 1][blocks]
    double* npart;             // [blocks]
    double2* xbuf;             // [2][N] vectors before their scaling (with the map inside)
    double *alpha, *beta;      // [m]
    double keep;               // second Gram-Schmidt pass when less than this share of |w|^2 is left
    unsigned* bar;             // [2] zero between launches
    int* err;                  // set when a barrier gave up
    const int64_t* row_ptr;    // hit records or CSR
    const uint2* hit;
    const double2 *amp, *dg;   // term amplitudes at u; diagonal sums, A and B parts
    double u;
    int has_b;
    const int32_t* col;
    const double2* val;
};

// Cooperative steps have the separate kernels to fall back on: a plan that does not fit, a launch that the
// driver refuses (fewer SMs for this process than the device has) and a grid barrier that gave up all end
// there, the last with the steps since the basis was last whole run again.  MOMED_COOP=0 starts there;
// =2 and =3 make every launch give up or be refused (tests).
enum CoopSwitch : int { COOP_OFF = 0, COOP_ON = 1, COOP_GIVES_UP = 2, COOP_REFUSED = 3 };
inline CoopSwitch coop_switch() {
    const char* e = std::getenv("MOMED_COOP");
    return e && (e[0] == '0' || e[0] == '2' || e[0] == '3') ? (CoopSwitch)(e[0] - '0') : COOP_ON;
}

// A cooperative launch, counted; false when the driver cannot hold the grid at once.
inline bool launch_cooperative(const void* k, int grid, int threads, void** args, size_t smem, cudaStream_t st) {
    const cudaError_t e = coop_switch() == COOP_REFUSED
                              ? cudaErrorCooperativeLaunchTooLarge
                              : cudaLaunchCooperativeKernel(k, dim3(grid), dim3(threads), args, smem, st);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        cudaGetLastError();
        return false;
    }
    MOMED_CUDA_TRY(e);
    note_launches(1);
    return true;
}

// the barrier, its exits and the error flag of a solve's launches
inline void clear_barrier(unsigned* bar, cudaStream_t st) {
    MOMED_CUDA_TRY(cudaMemsetAsync(bar, 0, 3 * sizeof(unsigned), st));
    if (coop_switch() == COOP_GIVES_UP) MOMED_CUDA_TRY(cudaMemsetAsync(bar + 2, 1, sizeof(unsigned), st));
}

// Rows per block and the split of a block's work; false where a block's part of w does not fit.
template <typename VT> bool cycle_plan(int64_t N, int map, CycleArgs<VT>& a, int& grid);
template <typename VT> bool launch_cycle(CycleArgs<VT>& a, int map, int grid, cudaStream_t st);

// The buffers of a solve's launches (partial sums, barrier) beside those the solver owns.
template <typename VT> struct CycleBufs {
    CycleArgs<VT> a{};
    int grid = 0, map = CYCLE_NONE;
    DevBuf<double2> part, xbuf;
    DevBuf<double> npart;
    DevBuf<unsigned> bar;
    // false: the solver runs its separate kernels
    bool prepare(int64_t N, int kind, double* alpha, double* beta, double keep, cudaStream_t st) {
        if (!cycle_plan(N, kind, a, grid)) return false;
        map = kind;
        part.resize((size_t)grid * (kMaxCols + 1));
        npart.resize(grid);
        bar.resize(3);
        clear_barrier(bar.p, st);
        if (map != CYCLE_NONE) xbuf.resize((size_t)2 * N);
        a.part = part.p;
        a.npart = npart.p;
        a.xbuf = xbuf.p;
        a.alpha = alpha;
        a.beta = beta;
        a.keep = keep;
        a.bar = bar.p;
        a.err = reinterpret_cast<int*>(bar.p + 2);
        return true;
    }
    // false: refused, nothing was done
    bool steps(VT* V, int j0, int j1, cudaStream_t st) {
        a.V = V;
        a.j0 = j0;
        a.j1 = j1;
        return launch_cycle(a, map, grid, st);
    }
};

}  // namespace momed
