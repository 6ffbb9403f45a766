// Construction and verification of the basis lookup tables (see index.cuh).
#include <algorithm>
#include <climits>

#include "index.cuh"

namespace momed {

namespace {

// One pass over the basis: its OR, the places where it does not ascend, and for every split point
// L the range of popcounts of the low L bits and of the rest.  A warp reads 32 states at a time
// and hands them round; each lane follows the split points L = lane and lane + 32 (lane 0 also 64).
// One launch per split point, as before, read the basis up to 65 times: 28 launches of 15 us on a
// 174k-state sector, 31 of 50 us on 1.0M states; this takes 15 and 56 us.
struct BasisScan {
    unsigned long long bits_or, bad;
    int range[65][4];                 // lo_min, lo_max, hi_min, hi_max
};

__global__ void __launch_bounds__(256) k_basis_scan(const uint64_t* __restrict__ b, int64_t n, BasisScan* out) {
    __shared__ int s_rng[65][4];
    for (int e = threadIdx.x; e < 65 * 4; e += 256) s_rng[e / 4][e % 4] = (e & 1) ? 0 : 64;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t m0 = (1ull << lane) - 1ull, m1 = (1ull << (lane + 32)) - 1ull;     // L = lane, lane + 32
    int r[8] = {64, 0, 64, 0, 64, 0, 64, 0}, tmin = 64, tmax = 0;
    uint64_t acc = 0;
    unsigned long long bad = 0;
    const int64_t warps = (int64_t)gridDim.x * 8, w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    for (int64_t i0 = w * 32; i0 < n; i0 += warps * 32) {
        const int64_t i = i0 + lane;
        const uint64_t s = i < n ? b[i] : 0ull;
        if (i < n) {
            acc |= s;
            if (i > 0 && s <= b[i - 1]) ++bad;
        }
        const int cnt = (int)min((int64_t)32, n - i0);
        for (int k = 0; k < cnt; ++k) {
            const uint64_t v = __shfl_sync(0xffffffffu, s, k);
            const int t = __popcll(v), a = __popcll(v & m0), c = __popcll(v & m1);
            r[0] = min(r[0], a); r[1] = max(r[1], a); r[2] = min(r[2], t - a); r[3] = max(r[3], t - a);
            r[4] = min(r[4], c); r[5] = max(r[5], c); r[6] = min(r[6], t - c); r[7] = max(r[7], t - c);
            tmin = min(tmin, t); tmax = max(tmax, t);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q & 1) {
            atomicMax(&s_rng[lane][q], r[q]);
            atomicMax(&s_rng[lane + 32][q], r[q + 4]);
        } else {
            atomicMin(&s_rng[lane][q], r[q]);
            atomicMin(&s_rng[lane + 32][q], r[q + 4]);
        }
    }
    if (lane == 0) {                  // L = 64: everything low
        atomicMin(&s_rng[64][0], tmin);
        atomicMax(&s_rng[64][1], tmax);
        atomicMin(&s_rng[64][2], 0);
    }
    for (int o = 16; o > 0; o >>= 1) {
        acc |= __shfl_xor_sync(0xffffffffu, acc, o);
        bad += __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if (lane == 0) {
        if (acc) atomicOr(&out->bits_or, (unsigned long long)acc);
        if (bad) atomicAdd(&out->bad, bad);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 65 * 4; e += 256) {
        if (e & 1) atomicMax(&out->range[e / 4][e % 4], s_rng[e / 4][e % 4]);
        else atomicMin(&out->range[e / 4][e % 4], s_rng[e / 4][e % 4]);
    }
}

struct Tables {
    PartDesc hi, lo;
    const uint32_t* binom;
};

__device__ __forceinline__ uint32_t slot_of(uint64_t s, const PartDesc& d, const uint32_t* binom) {
    return part_slot(s, d, d.base, binom);
}

__global__ void k_build_off_hi(const uint64_t* __restrict__ b, int64_t n, Tables t, uint32_t* off_hi) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t hi = t.hi.width ? (b[i] >> t.hi.shift) : 0ull;
        uint64_t prev = (i > 0 && t.hi.width) ? (b[i - 1] >> t.hi.shift) : ~0ull;
        if (i == 0 || hi != prev) off_hi[slot_of(b[i], t.hi, t.binom)] = (uint32_t)i;
    }
}

__global__ void k_build_rank_lo(const uint64_t* __restrict__ b, int64_t n, Tables t, const uint32_t* off_hi,
                                uint32_t* rank_lo) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t o = off_hi[slot_of(b[i], t.hi, t.binom)];
        rank_lo[slot_of(b[i], t.lo, t.binom)] = (uint32_t)(i - (int64_t)o);
    }
}

__global__ void k_verify(const uint64_t* __restrict__ b, int64_t n, Tables t, const uint32_t* off_hi,
                         const uint32_t* rank_lo, unsigned long long* bad) {
    unsigned long long cnt = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (i > 0 && b[i] <= b[i - 1]) { ++cnt; continue; }     // must be strictly ascending
        int64_t j = (int64_t)off_hi[slot_of(b[i], t.hi, t.binom)] + (int64_t)rank_lo[slot_of(b[i], t.lo, t.binom)];
        if (j != i) ++cnt;
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(bad, cnt);
}

uint64_t host_binom(int n, int k) {
    if (k < 0 || k > n) return 0;
    uint64_t r = 1;
    for (int i = 1; i <= k; ++i) r = r * (uint64_t)(n - k + i) / (uint64_t)i;
    return r;
}

// Fill a part descriptor for bits [shift, shift + width) with popcounts in [cmin, cmax];
// returns table entries (UINT64_MAX when the part cannot be tabulated).
uint64_t plan_part(PartDesc& d, int shift, int width, int cmin, int cmax) {
    d = PartDesc{};
    d.shift = shift;
    d.width = width;
    d.cmin = cmin;
    d.cmax = cmax;
    if (width == 0) { d.mode = PART_DIRECT; d.size = 1; return 1; }
    uint64_t direct = width <= 26 ? (1ull << width) : UINT64_MAX;
    uint64_t comb = UINT64_MAX;
    if (width <= 32 && cmin <= cmax) {
        comb = 0;
        for (int c = cmin; c <= cmax; ++c) comb += host_binom(width, c);
    }
    // combinadic costs a few instructions per set bit: take it only when it shrinks the table 2x
    if (comb != UINT64_MAX && (direct == UINT64_MAX || comb * 2 <= direct)) {
        d.mode = PART_COMBINADIC;
        uint64_t acc = 0;
        for (int c = cmin; c <= cmax; ++c) { d.base[c - cmin] = (uint32_t)acc; acc += host_binom(width, c); }
        d.size = (uint32_t)comb;
        return comb;
    }
    if (direct == UINT64_MAX) return UINT64_MAX;
    d.mode = PART_DIRECT;
    d.size = (uint32_t)direct;
    return direct;
}

int grid_for(int64_t n, int threads = 256) {
    int64_t blocks = (n + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, 148 * 16));
}

}  // namespace

// Table size cap: 2^26 entries per table (256 MiB as uint32).
static constexpr uint64_t kMaxTableEntries = 1ull << 26;

// The basis facts the index plan and the handle need (basis_or, whether it ascends, popcount
// ranges), in one launch and one copy.
void scan_basis(momed_handle* h) {
    BasisScan init{};
    for (auto& r : init.range) { r[0] = 64; r[1] = 0; r[2] = 64; r[3] = 0; }
    BasisScan got = init;
    if (h->n > 0) {
        cudaStream_t st = h->stream;
        h->scan.resize(sizeof(BasisScan));
        BasisScan* d = reinterpret_cast<BasisScan*>(h->scan.p);
        MOMED_CUDA_TRY(cudaMemcpyAsync(d, &init, sizeof(init), cudaMemcpyHostToDevice, st));
        // two batches of 32 states per warp, up to the resident blocks (every further block adds a
        // merge of its 65 x 4 ranges)
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((h->n + 511) / 512, 148 * 8));
        k_basis_scan<<<grid, 256, 0, st>>>(h->basis.p, h->n, d);
        MOMED_CUDA_TRY(cudaGetLastError());
        note_launches(1);
        MOMED_CUDA_TRY(cudaMemcpyAsync(&got, d, sizeof(got), cudaMemcpyDeviceToHost, st));
        MOMED_CUDA_TRY(cudaStreamSynchronize(st));
    }
    h->basis_or = got.bits_or;
    h->basis_bad = (int64_t)got.bad;
    std::copy(&got.range[0][0], &got.range[0][0] + 65 * 4, h->basis_range);
    h->basis_pop_max = h->n > 0 ? got.range[0][3] : 0;       // at L = 0 the high part is the whole state
    h->basis_scanned = true;
}

void build_index(momed_handle* h) {
    Index& ix = h->index;
    ix.mode = INDEX_SEARCH;
    ix.misses_checked = -1;
    const int64_t n = h->n;
    cudaStream_t st = h->stream;
    if (n == 0) return;
    MOMED_REQUIRE(n < (int64_t)kInvalid, MOMED_EINVAL, "basis larger than 2^32-1 states");
    if (!h->basis_scanned) scan_basis(h);
    MOMED_REQUIRE(h->basis_bad == 0, MOMED_EINVAL, "basis must be sorted ascending without duplicates");
    h->counters.resize(16);
    unsigned long long* dc = h->counters.p;
    uint64_t bits_or = h->basis_or | h->op_mask_or;
    int nbits = bits_or ? 64 - __builtin_clzll(bits_or) : 1;
    const int* ranges = h->basis_range;       // popcount ranges for every split point

    // choose the split minimising table entries; widen popcount ranges by the largest
    // change a term can make so that every target of a hit maps into the tables
    int best_L = -1;
    uint64_t best = UINT64_MAX;
    PartDesc best_hi{}, best_lo{};
    for (int L = 0; L <= nbits; ++L) {
        PartDesc lo, hi;
        int lomin = ranges[4 * L], lomax = ranges[4 * L + 1], himin = ranges[4 * L + 2], himax = ranges[4 * L + 3];
        uint64_t slo = plan_part(lo, 0, L, lomin, lomax);
        uint64_t shi = plan_part(hi, L, nbits - L, himin, himax);
        if (slo == UINT64_MAX || shi == UINT64_MAX) continue;
        if (slo > kMaxTableEntries || shi > kMaxTableEntries) continue;
        uint64_t tot = slo + shi;
        if (tot < best) { best = tot; best_L = L; best_hi = hi; best_lo = lo; }
    }
    ix.hi = best_hi;
    ix.lo = best_lo;
    if (best_L < 0) return;   // search mode

    ix.off_hi.resize(ix.hi.size);
    ix.rank_lo.resize(ix.lo.size);
    MOMED_CUDA_TRY(cudaMemsetAsync(ix.off_hi.p, 0xFF, (size_t)ix.hi.size * 4, st));
    MOMED_CUDA_TRY(cudaMemsetAsync(ix.rank_lo.p, 0xFF, (size_t)ix.lo.size * 4, st));
    Tables t{ix.hi, ix.lo, h->binom.p};
    k_build_off_hi<<<grid_for(n), 256, 0, st>>>(h->basis.p, n, t, ix.off_hi.p);
    k_build_rank_lo<<<grid_for(n), 256, 0, st>>>(h->basis.p, n, t, ix.off_hi.p, ix.rank_lo.p);
    MOMED_CUDA_TRY(cudaMemsetAsync(dc + 2, 0, sizeof(unsigned long long), st));
    k_verify<<<grid_for(n), 256, 0, st>>>(h->basis.p, n, t, ix.off_hi.p, ix.rank_lo.p, dc + 2);
    unsigned long long bad = 0;
    MOMED_CUDA_TRY(cudaMemcpyAsync(&bad, dc + 2, sizeof(bad), cudaMemcpyDeviceToHost, st));
    MOMED_CUDA_TRY(cudaStreamSynchronize(st));
    if (bad == 0) {
        ix.mode = INDEX_CHECKED;   // promoted to RANKED once an operator validates without misses
    } else {
        ix.off_hi.release();
        ix.rank_lo.release();
        ix.mode = INDEX_SEARCH;
    }
}

IndexView index_view(const momed_handle* h) {
    IndexView v{};
    v.basis = h->basis.p;
    v.n = h->n;
    v.off_hi = h->index.off_hi.p;
    v.rank_lo = h->index.rank_lo.p;
    v.hi = h->index.hi;
    v.lo = h->index.lo;
    v.mode = h->index.mode;
    v.binom = h->binom.p;
    return v;
}

}  // namespace momed
