// One step of the lockstep block Lanczos (batch.cu) beside its map, as one cooperative launch
// (blockstep.cu), and the 16-byte packets in which the block kernels read their vectors.
#pragma once
#include "cycle.cuh"

namespace momed {

// 16-byte packets of a block vector: two c64 values (adjacent right-hand sides of one row) when
// NB is even, else one value.
template <typename VT, int NB> struct Pack {
    static constexpr int E = 1;
    using T = VT;
    static __device__ __forceinline__ void get(const T& p, double2* v) { v[0] = to_d2(p); }
    static __device__ __forceinline__ T put(const double2* v) { return from_d2<VT>(v[0]); }
};
template <int NB> struct PackF2 {
    static constexpr int E = 2;
    using T = float4;
    static __device__ __forceinline__ void get(const float4& p, double2* v) {
        v[0] = make_double2(p.x, p.y);
        v[1] = make_double2(p.z, p.w);
    }
    static __device__ __forceinline__ float4 put(const double2* v) {
        return make_float4((float)v[0].x, (float)v[0].y, (float)v[1].x, (float)v[1].y);
    }
};
template <> struct Pack<float2, 2> : PackF2<2> {};
template <> struct Pack<float2, 4> : PackF2<4> {};
template <> struct Pack<float2, 8> : PackF2<8> {};
template <> struct Pack<float2, 16> : PackF2<16> {};
template <> struct Pack<float2, 32> : PackF2<32> {};

// Block vectors x[row * NB + r]; column i of the basis at V + i N NB.
template <typename VT> struct BlockStepArgs {
    VT* V;
    int64_t N;
    int j, m;                  // the step: column j + 1 (the map's result) against columns [0, j]
    int rows;                  // rows per block
    double2* part;             // [(m + 1) NB][blocks]
    double2* coef;             // [(m + 1) NB]
    double* npart;             // [blocks][NB]
    double *alpha, *beta;      // [NB][m]
    double keep;               // second Gram-Schmidt pass when less than this share of |w|^2 is left
    unsigned* bar;             // [2] zero between launches
    int* err;                  // set when a barrier gave up
};

// Rows per block and the grid for bases of m + 1 columns; false where a launch cannot be resident.
template <typename VT> bool block_step_plan(int64_t N, int nb, int m, BlockStepArgs<VT>& a, int& grid);
template <typename VT> bool launch_block_step(const BlockStepArgs<VT>& a, int nb, int grid, cudaStream_t st);

template <typename VT> struct BlockStepBufs {
    BlockStepArgs<VT> a{};
    int nb = 0, grid = 0;
    DevBuf<double2> part, coef;
    DevBuf<double> npart;
    DevBuf<unsigned> bar;
    bool prepare(int64_t N, int nrhs, int m, double* alpha, double* beta, cudaStream_t st) {
        if (!block_step_plan(N, nrhs, m, a, grid)) return false;
        nb = nrhs;
        part.resize((size_t)grid * (m + 1) * nb);
        coef.resize((size_t)(m + 1) * nb);
        npart.resize((size_t)grid * nb);
        bar.resize(3);
        clear_barrier(bar.p, st);
        a.m = m;
        a.part = part.p;
        a.coef = coef.p;
        a.npart = npart.p;
        a.alpha = alpha;
        a.beta = beta;
        a.bar = bar.p;
        a.err = reinterpret_cast<int*>(bar.p + 2);
        return true;
    }
    // false: refused, nothing was done
    bool step(VT* V, int j, double keep, cudaStream_t st) {
        a.V = V;
        a.j = j;
        a.keep = keep;
        return launch_block_step(a, nb, grid, st);
    }
};

}  // namespace momed
