// Analysis of eigenvectors on the device: the one-body reduced density matrix and the
// many-body connection step of the quantum-geometry analysis.
//
// Reference: PES_1rdm (MomentumED/src/analysis/particle_reduced_density_matrix.jl:4-33):
// rdm[i][j] = <psi| c+_i c_j |psi> for i <= j, summed over basis states x_in with j occupied,
// mid = x_in - j, i empty in mid (or i = j), x_out = mid + i found in the subspace (index_fit),
// sign (-1)^(scat_occ_number(mid, i) + scat_occ_number(mid, j)) where scat_occ_number counts
// the occupied orbitals above the given one; then rdm[i][j] = conj(rdm[j][i]) for i > j.
//
// One thread per basis state walks its occupied orbitals j and the empty orbitals i < j; targets are
// looked up with key checks (c+_i c_j usually leaves a momentum sector), and those in the basis add to
// the block's norb x norb matrix in shared memory.  The occupations (i = j), which every state has,
// are summed across the warp orbital by orbital instead: as shared-memory atomics, all lanes on the
// same few diagonal elements, they took most of the kernel (345 us on a 174k-state sector of 27
// orbitals, 163 without them).  What is left waits for the lookups' table reads, so three blocks of 16
// warps share an SM (126 us; two of 8 before).  A second kernel adds the blocks' matrices (the host
// did, after copying all of them: 3.4 MB).
#include "candidates.cuh"

namespace momed {

namespace {

constexpr int kRdmThreads = 256;
constexpr int kRdm1Threads = 512;

__global__ void __launch_bounds__(kRdm1Threads)
k_rdm1(IndexView iv, const double2* __restrict__ psi, int norb, double2* __restrict__ partial) {
    extern __shared__ double2 acc[];                  // [norb * norb]
    __shared__ SharedTables sh;
    const int nn = norb * norb;
    for (int e = threadIdx.x; e < nn; e += blockDim.x) acc[e] = make_double2(0.0, 0.0);
    stage_tables(sh, iv);                             // ends with __syncthreads
    const uint64_t omask = norb >= 64 ? ~0ull : ((1ull << norb) - 1ull);
    const int lane = threadIdx.x & 31;
    double occ0 = 0.0, occ1 = 0.0;                    // occupations of orbitals lane and lane + 32
    for (int64_t x0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); x0 < iv.n;
         x0 += (int64_t)gridDim.x * blockDim.x) {     // warp-uniform
        const int64_t x = x0 + lane;
        const bool in = x < iv.n;
        const uint64_t s = in ? __ldg(iv.basis + x) : 0ull;
        const double2 pin = in ? __ldg(psi + x) : make_double2(0.0, 0.0);
        const double p2 = pin.x * pin.x + pin.y * pin.y;
        for (int o = 0; o < norb; ++o) {
            const bool has = (s >> o) & 1ull;
            if (!__any_sync(kFull, has)) continue;
            double v = has ? p2 : 0.0;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
            if (lane == (o & 31)) {
                if (o < 32) occ0 += v;
                else occ1 += v;
            }
        }
        uint64_t rem = s & omask;
        while (rem) {
            const int j = __ffsll((long long)rem) - 1;
            rem &= rem - 1ull;
            const uint64_t mid = s & ~(1ull << j);
            const uint64_t above_j = j >= 63 ? 0ull : (~0ull << (j + 1));
            for (uint64_t free = ~mid & ((1ull << j) - 1ull); free; free &= free - 1ull) {
                const int i = __ffsll((long long)free) - 1;
                const int64_t y = lookup_index(iv, mid | (1ull << i), sh.base_hi, sh.base_lo, sh.binom);
                if (y < 0) continue;
                const uint64_t above_i = ~0ull << (i + 1);              // i < j <= 63
                const bool neg = ((__popcll(mid & above_i) + __popcll(mid & above_j)) & 1) != 0;
                const double2 pout = __ldg(psi + y);
                double vr = pout.x * pin.x + pout.y * pin.y;      // conj(psi[y]) * psi[x]
                double vi = pout.x * pin.y - pout.y * pin.x;
                if (neg) { vr = -vr; vi = -vi; }
                atomicAdd(&acc[i * norb + j].x, vr);
                atomicAdd(&acc[i * norb + j].y, vi);
            }
        }
    }
    if (lane < norb) atomicAdd(&acc[lane * norb + lane].x, occ0);
    if (lane + 32 < norb) atomicAdd(&acc[(lane + 32) * norb + lane + 32].x, occ1);
    __syncthreads();
    for (int e = threadIdx.x; e < nn; e += blockDim.x) partial[(int64_t)blockIdx.x * nn + e] = acc[e];
}

// out[e] = sum over the blocks of partial[b][e]: a warp per element, its lanes over the blocks in a
// fixed stride and tree
__global__ void k_sum_blocks(const double2* __restrict__ partial, int blocks, int count, double2* __restrict__ out) {
    const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (e >= count) return;
    double2 s = make_double2(0.0, 0.0);
    for (int b = lane; b < blocks; b += 32) {
        const double2 v = __ldg(partial + (int64_t)b * count + e);
        s.x += v.x;
        s.y += v.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(kFull, s.x, o);
        s.y += __shfl_xor_sync(kFull, s.y, o);
    }
    if (lane == 0) out[e] = s;
}

// ED_step_inner_prod (MomentumED/src/analysis/manybody_quantum_geometry.jl:48-94): thread per
// basis state; the product of the orbital overlaps over its occupied orbitals (ascending, as
// occ_list gives them), then conj(psi_f[j][x]) psi_i[k][x] times that product for every (j, k),
// accumulated per block in shared memory (g <= 32).
__global__ void __launch_bounds__(kRdmThreads)
k_step_inner(const uint64_t* __restrict__ basis, int64_t n, const double2* __restrict__ psi_f,
             const double2* __restrict__ psi_i, int g, const double2* __restrict__ orb, int norb,
             double2* __restrict__ partial) {
    extern __shared__ double2 acc[];                  // [g * g]
    __shared__ double2 s_orb[64];
    const int gg = g * g;
    for (int e = threadIdx.x; e < gg; e += blockDim.x) acc[e] = make_double2(0.0, 0.0);
    if (threadIdx.x < 64) s_orb[threadIdx.x] = threadIdx.x < norb ? orb[threadIdx.x] : make_double2(1.0, 0.0);
    __syncthreads();
    const uint64_t omask = norb >= 64 ? ~0ull : ((1ull << norb) - 1ull);
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
        uint64_t rem = __ldg(basis + x) & omask;
        double pr = 1.0, pi = 0.0;
        while (rem) {
            const int o = __ffsll((long long)rem) - 1;
            rem &= rem - 1ull;
            const double2 w = s_orb[o];
            const double r = pr * w.x - pi * w.y, i = pr * w.y + pi * w.x;
            pr = r;
            pi = i;
        }
        for (int j = 0; j < g; ++j) {
            const double2 f = __ldg(psi_f + (int64_t)j * n + x);
            for (int k = 0; k < g; ++k) {
                const double2 v = __ldg(psi_i + (int64_t)k * n + x);
                const double cr = f.x * v.x + f.y * v.y, ci = f.x * v.y - f.y * v.x;   // conj(f) * v
                atomicAdd(&acc[j * g + k].x, cr * pr - ci * pi);
                atomicAdd(&acc[j * g + k].y, cr * pi + ci * pr);
            }
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < gg; e += blockDim.x) partial[(int64_t)blockIdx.x * gg + e] = acc[e];
}

}  // namespace

void step_inner_prod(momed_handle* h, const double* psi_f, const double* psi_i, int g, const double* orb, int norb,
                     double* out) {
    MOMED_REQUIRE(g >= 1 && g <= 32, MOMED_EINVAL, "g must be in [1, 32]");
    MOMED_REQUIRE(norb >= 1 && norb <= 64, MOMED_EINVAL, "norb must be in [1, 64]");
    MOMED_REQUIRE(!h->sparse_only && h->n > 0, MOMED_ESTATE, "set a basis first (momed_set_basis)");
    MOMED_REQUIRE(norb == 64 || (h->basis_or >> norb) == 0, MOMED_EINVAL, "basis states use orbitals beyond norb");
    const int64_t n = h->n;
    cudaStream_t st = h->stream;
    DevBuf<double2> fd, id, od, part;
    fd.resize((size_t)g * n);
    id.resize((size_t)g * n);
    od.resize(norb);
    MOMED_CUDA_TRY(cudaMemcpyAsync(fd.p, psi_f, (size_t)g * n * 16, cudaMemcpyHostToDevice, st));
    MOMED_CUDA_TRY(cudaMemcpyAsync(id.p, psi_i, (size_t)g * n * 16, cudaMemcpyHostToDevice, st));
    MOMED_CUDA_TRY(cudaMemcpyAsync(od.p, orb, (size_t)norb * 16, cudaMemcpyHostToDevice, st));
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + kRdmThreads - 1) / kRdmThreads, (int64_t)sms * 2));
    const int gg = g * g;
    part.resize((size_t)grid * gg);
    k_step_inner<<<grid, kRdmThreads, (size_t)gg * sizeof(double2), st>>>(h->basis.p, n, fd.p, id.p, g, od.p, norb,
                                                                          part.p);
    MOMED_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    DevBuf<double2> sum;
    sum.resize(gg);
    k_sum_blocks<<<(gg + 7) / 8, 256, 0, st>>>(part.p, grid, gg, sum.p);
    MOMED_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    MOMED_CUDA_TRY(cudaMemcpyAsync(out, sum.p, (size_t)gg * 16, cudaMemcpyDeviceToHost, st));
    MOMED_CUDA_TRY(cudaStreamSynchronize(st));
}

void rdm1(momed_handle* h, const double* psi, int norb, double* rdm) {
    MOMED_REQUIRE(norb >= 1 && norb <= 64, MOMED_EINVAL, "norb must be in [1, 64]");
    MOMED_REQUIRE(!h->sparse_only && h->n > 0, MOMED_ESTATE, "set a basis first (momed_set_basis)");
    MOMED_REQUIRE(norb == 64 || (h->basis_or >> norb) == 0, MOMED_EINVAL, "basis states use orbitals beyond norb");
    if (h->index_dirty || (h->op_mask_or & ~h->index_bits)) {
        h->index_bits = h->basis_or | h->op_mask_or;
        build_index(h);
        h->index_dirty = false;
        h->op_validated = false;
    }
    IndexView iv = index_view(h);
    if (iv.mode == INDEX_RANKED) iv.mode = INDEX_CHECKED;     // targets leave the sector: compare keys
    const int64_t n = h->n;
    cudaStream_t st = h->stream;
    DevBuf<double2> pd, part;
    pd.resize(n);
    MOMED_CUDA_TRY(cudaMemcpyAsync(pd.p, psi, n * 16, cudaMemcpyHostToDevice, st));
    const int nn = norb * norb;
    const size_t smem = (size_t)nn * sizeof(double2);
    constexpr size_t smem_max = 64 * 64 * sizeof(double2);
    // process-wide kernel attribute: always the largest size, so concurrent callers never lower it
    MOMED_CUDA_TRY(cudaFuncSetAttribute(k_rdm1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + kRdm1Threads - 1) / kRdm1Threads, (int64_t)sms * 3));
    part.resize((size_t)grid * nn);
    k_rdm1<<<grid, kRdm1Threads, smem, st>>>(iv, pd.p, norb, part.p);
    MOMED_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    DevBuf<double2> sum;
    sum.resize(nn);
    k_sum_blocks<<<(nn + 7) / 8, 256, 0, st>>>(part.p, grid, nn, sum.p);
    MOMED_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    MOMED_CUDA_TRY(cudaMemcpyAsync(rdm, sum.p, (size_t)nn * 16, cudaMemcpyDeviceToHost, st));
    MOMED_CUDA_TRY(cudaStreamSynchronize(st));
    for (int i = 0; i < norb; ++i)
        for (int j = 0; j < i; ++j) {
            rdm[2 * ((size_t)i * norb + j)] = rdm[2 * ((size_t)j * norb + i)];
            rdm[2 * ((size_t)i * norb + j) + 1] = -rdm[2 * ((size_t)j * norb + i) + 1];
        }
}

}  // namespace momed
