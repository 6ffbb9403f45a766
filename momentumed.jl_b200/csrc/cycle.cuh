// Cooperative kernels for Lanczos steps: a single-vector cycle (cycle.cu), a step of the lockstep block
// solver (blockstep.cu).
#pragma once
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

// Rows per block and the split of a block's work; false where a block's part of w does not fit.
template <typename VT> bool cycle_plan(int64_t N, CycleArgs<VT>& a, int& grid);
template <typename VT> void launch_cycle(CycleArgs<VT>& a, int map, int grid, cudaStream_t st);

// The buffers of a solve's launches (partial sums, barrier) beside those the solver owns.
template <typename VT> struct CycleBufs {
    CycleArgs<VT> a{};
    int grid = 0;
    DevBuf<double2> part, xbuf;
    DevBuf<double> npart;
    DevBuf<unsigned> bar;
    // false: the solver runs its separate kernels
    bool prepare(int64_t N, bool with_map, double* alpha, double* beta, double keep, cudaStream_t st) {
        if (!cycle_plan(N, a, grid)) return false;
        part.resize((size_t)grid * (kMaxCols + 1));
        npart.resize(grid);
        bar.resize(3);                   // barrier, its exits, the error flag
        MOMED_CUDA_TRY(cudaMemsetAsync(bar.p, 0, 3 * sizeof(unsigned), st));
        if (with_map) xbuf.resize((size_t)2 * N);
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
    void steps(VT* V, int j0, int j1, int map, cudaStream_t st) {
        a.V = V;
        a.j0 = j0;
        a.j1 = j1;
        launch_cycle(a, map, grid, st);
    }
    // after a synchronisation of the copy of err: a barrier that gave up ends the solve
    static void check(int err) {
        if (err) throw Error{MOMED_ETIMEOUT, "Lanczos cycle: a grid barrier gave up"};
    }
};

}  // namespace momed
