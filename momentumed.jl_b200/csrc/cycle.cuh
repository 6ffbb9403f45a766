// Cooperative kernel for the steps of an FP64 Lanczos cycle (cycle.cu).
#pragma once
#include "vecops.cuh"

namespace momed {

enum CycleMap : int { CYCLE_NONE = 0, CYCLE_HITS = 1, CYCLE_CSR = 2 };

struct CycleArgs {
    double2* V;                // basis, column i at V + i N
    int64_t N;
    int j0, j1;                // steps [j0, j1); column j0 is normalised
    int rows, chunks, split;   // cycle_plan
    double2* part;             // [kMaxCols + 1][blocks]
    double* npart;             // [blocks]
    double2* xbuf;             // [2][N] vectors before their scaling (with the map inside)
    double *alpha, *beta;      // [m]
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

bool cycle_plan(int64_t N, CycleArgs& a, int& grid);
void launch_cycle(CycleArgs& a, int map, int grid, cudaStream_t st);

}  // namespace momed
