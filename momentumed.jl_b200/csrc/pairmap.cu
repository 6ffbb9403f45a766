// Pair-factorised form of the matrix-free map, one right-hand side.
//
// The two-body part of H acts through pair operators: H2 = sum over pair classes of
// sum_pq V[p][q] P+_p P_q, where a class is a set of orbital pairs that the term list couples
// (for a momentum-conserving interaction the pairs of one total momentum and particle content).
// ka_linearmap_kernel! (MomentumED/src/method/gpu_interface.jl:128-163) and the hit cache
// (hitcache.cu) visit every (row, term) hit, n * ~hits_per_row gathers of x.  Here the product is
// taken in two steps through the states with two particles removed:
//
//   phi_q(s')  = sign(s', q) x[s' + q]           for every pair q of the class free in s'
//   psi_p(s')  = sum_q V[p][q] phi_q(s')         (a dense P x P product per s', P = pairs of a class;
//                                                 V[p][p] = 0: a pair with itself is of the diagonal)
//   y[s]       = sum over pairs p of s of sign(s - p, p) psi_p(s - p)  + diagonal[s] x[s]
//
// The fermionic sign of a term factorises over its two pairs: popcount(s' & (pm_out ^ pm_in)) is
// even exactly when those of its two masks agree.  A row has Ne (Ne - 1) / 2 pairs, so a map
// gathers n Ne (Ne - 1) / 2 values twice (x, then psi) where the hit cache gathers one value for
// each hit: 6.2M + 6.2M against 38.2M on a 3x9 Ne = 9 sector, 132M + 132M against 1.8G on the
// two-component 4x6 one, and stores 8 bytes per (row, pair) entry instead of 8 per hit.
//
// Tables (built once per basis and operator; entry = one (row, pair) with the pair in a class):
//   ids        intermediate states in class-major order, 32 per tile (classes padded to a tile),
//              sorted in windows within a class
//   tile[t]    {pairs of the class that some state of the tile has free and that lead to a basis
//              state, first slot, first entry}
//   ent_row[slot]    row of s' + q, sign in bit 31; ~0 where the state has no such entry.  A tile
//              has 32 slots for each of its pairs, so a warp's reads are runs of 32 values at a
//              constant step without any bit counting
//   psi[e]     workspace, one value per entry: for each pair of a tile the lanes that have it,
//              packed.  With a value per slot (1.5x as many) psi of a 3x9 sector left the L2: the
//              row kernel took 44 us instead of 33 in FP64, 25 instead of 18 in FP32
//   row_ent[k][row]  entry of the row's k-th pair (pairs counted from the highest orbitals, which
//              neighbouring rows share, so their psi values are neighbours)
// Slot and entry ranges follow atomic counters, so the tables can differ from build to build; every value
// of psi and the order of every sum is fixed, so the product is the same to the bit.
#include <algorithm>
#include <chrono>
#include <cstdlib>
#include <numeric>
#include <string>
#include <type_traits>

#include "candidates.cuh"

namespace momed {

namespace {

constexpr int kMaxClassPairs = 32;      // one availability bit per pair
constexpr int kMaxClasses = 2048;       // per-block class counters in shared memory
constexpr uint32_t kNoEntry = 0xFFFFFFFFu;
constexpr int kPT = 256;                // threads of the build and row kernels
constexpr int kIdWarps = 4;             // warps of a k_pair_ids block

// bits strictly between the two orbitals of a pair mask
__host__ __device__ __forceinline__ uint64_t between(uint64_t m) {
#ifdef __CUDA_ARCH__
    const int lo = __ffsll((long long)m) - 1, hi = 63 - __clzll((long long)m);
#else
    const int lo = __builtin_ctzll(m), hi = 63 - __builtin_clzll(m);
#endif
    return ((1ull << hi) - 1ull) & ~((2ull << lo) - 1ull);
}

// occupied orbitals of s above orbital a
__device__ __forceinline__ int above(uint64_t s, int a) { return a >= 63 ? 0 : __popcll(s >> (a + 1)); }

// l-th occupied orbital from the top
__device__ __forceinline__ int from_top(uint64_t s, int l) {
    for (; l > 0; --l) s &= ~(1ull << (63 - __clzll((long long)s)));
    return 63 - __clzll((long long)s);
}

// s minus its k-th pair (u < v from the top, k = v (v - 1) / 2 + u) and that pair's class and slot
// (-1: no such pair, or a pair that no term names)
__device__ __forceinline__ int pair_at(uint64_t s, int ne, int k, const int32_t* __restrict__ ptab, uint64_t& rest) {
    int u, v;
    pair_of(k, u, v);
    if (v >= ne) return -1;
    const int hi = from_top(s, u), lo = from_top(s, v);
    rest = s & ~(1ull << hi) & ~(1ull << lo);
    return __ldg(ptab + lo * 64 + hi);
}

// table reads of a map: each value once, so not kept in L1 (3% of a map)
__device__ __forceinline__ uint32_t ld_stream(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// own[k][row] = 1 where the row is the first basis state of the intermediate state: no earlier
// pair of the class leads to one.  counts[class][block]: owners per class.
__global__ void __launch_bounds__(kPT)
k_pair_own(IndexView iv, PairPlanView pp, int kmax, int64_t rows_per_block, uint8_t* __restrict__ own,
           int32_t* __restrict__ counts) {
    __shared__ SharedTables sh;
    extern __shared__ int hist[];
    for (int c = threadIdx.x; c < pp.nclass; c += kPT) hist[c] = 0;
    stage_tables(sh, iv);                                     // ends with __syncthreads
    const int64_t r0 = (int64_t)blockIdx.x * rows_per_block, r1 = min(iv.n, r0 + rows_per_block);
    const uint32_t nr = r1 > r0 ? (uint32_t)(r1 - r0) : 0u;
    for (uint32_t it = threadIdx.x; it < nr * (uint32_t)kmax; it += kPT) {
        const int64_t row = r0 + it % nr;
        const int k = (int)(it / nr);
        const uint64_t s = __ldg(iv.basis + row);
        uint64_t rest = 0;
        const int cs = pair_at(s, __popcll(s), k, pp.ptab, rest);
        bool mine = cs >= 0;
        if (mine) {
            const int4 cl = __ldg(pp.cls + (cs >> 8));
            for (int q = 0; q < (cs & 255) && mine; ++q) {
                const uint64_t m = __ldg(pp.mask + cl.y + q);
                if ((rest & m) == 0 && lookup_index(iv, rest | m, sh.base_hi, sh.base_lo, sh.binom) >= 0) mine = false;
            }
            if (mine) atomicAdd(&hist[cs >> 8], 1);
        }
        own[(int64_t)k * iv.n + row] = mine ? 1 : 0;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < pp.nclass; c += kPT) counts[(int64_t)c * gridDim.x + blockIdx.x] = hist[c];
}

// exclusive sums over the blocks of each class (one warp per class), totals per class
__global__ void k_pair_scan(int32_t* __restrict__ counts, int nblk, int nclass, int32_t* __restrict__ total) {
    const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= nclass) return;
    int run = 0;
    for (int b0 = 0; b0 < nblk; b0 += 32) {
        const int b = b0 + lane;
        const int v = b < nblk ? counts[(int64_t)c * nblk + b] : 0;
        int incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        if (b < nblk) counts[(int64_t)c * nblk + b] = run + incl - v;
        run += __shfl_sync(kFull, incl, 31);
    }
    if (lane == 0) total[c] = run;
}

// ids of the owned intermediate states
__global__ void __launch_bounds__(kPT)
k_pair_assign(IndexView iv, PairPlanView pp, int kmax, int64_t rows_per_block, const uint8_t* __restrict__ own,
              const int32_t* __restrict__ offs, const int32_t* __restrict__ cbase, uint64_t* __restrict__ sp) {
    extern __shared__ int hist[];
    for (int c = threadIdx.x; c < pp.nclass; c += kPT)
        hist[c] = __ldg(cbase + c) + offs[(int64_t)c * gridDim.x + blockIdx.x];
    __syncthreads();
    const int64_t r0 = (int64_t)blockIdx.x * rows_per_block, r1 = min(iv.n, r0 + rows_per_block);
    const uint32_t nr = r1 > r0 ? (uint32_t)(r1 - r0) : 0u;
    for (uint32_t it = threadIdx.x; it < nr * (uint32_t)kmax; it += kPT) {
        const int64_t row = r0 + it % nr;
        const int k = (int)(it / nr);
        if (!own[(int64_t)k * iv.n + row]) continue;
        const uint64_t s = __ldg(iv.basis + row);
        uint64_t rest = 0;
        const int cs = pair_at(s, __popcll(s), k, pp.ptab, rest);
        sp[atomicAdd(&hist[cs >> 8], 1)] = rest;
    }
}

// Sorts the states of a class in windows of kSortIds (bitonic, in shared memory): neighbouring ids
// then share their high orbitals, so the pairs that are free and the rows they lead to agree
// between the lanes of a tile.  On a 3x9 sector (counted on the tables): 0.54 -> 0.43 cache lines
// of x per entry, 0.47 -> 0.39 of psi, 11.2 -> 10.7 pairs of 13 that any lane of a tile has; a full
// sort would give 0.38 and 0.36.
constexpr int kSortIds = 4096;
__global__ void __launch_bounds__(1024)
k_pair_sort(const int2* __restrict__ win, uint64_t* __restrict__ sp) {
    __shared__ uint64_t key[kSortIds];
    const int2 w = __ldg(win + blockIdx.x);                   // {first id, ids}
    for (int i = threadIdx.x; i < kSortIds; i += 1024) key[i] = i < w.y ? sp[(int64_t)w.x + i] : ~0ull;
    int len = 2;
    while (len < w.y) len <<= 1;                              // power of two that holds the window
    for (int size = 2; size <= len; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int i = threadIdx.x; i < len / 2; i += 1024) {
                const int a = 2 * i - (i & (stride - 1)), b = a + stride;
                const uint64_t x = key[a], y = key[b];
                if ((x > y) == ((a & size) == 0)) {
                    key[a] = y;
                    key[b] = x;
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < w.y; i += 1024) sp[(int64_t)w.x + i] = key[i];
}

// The slots of every tile (one warp per tile): tile, ent_row and its transpose row_ent.  tot[0]
// counts entries, tot[1] off-diagonal (row, term) hits, tot[2] and tot[4] hand out the tiles'
// slot and entry ranges, tot[3] counts entries that fell outside the tables (never written).  Padding ids have the state
// ~0: no pair is free in it.
__global__ void __launch_bounds__(kIdWarps * 32)
k_pair_fill(IndexView iv, PairPlanView pp, const int4* __restrict__ work, const uint64_t* __restrict__ sp,
            uint4* __restrict__ tile, uint32_t* __restrict__ ent_row, uint32_t* __restrict__ row_ent, int kmax,
            unsigned long long nslot, unsigned long long nent, unsigned long long* __restrict__ tot) {
    __shared__ SharedTables sh;
    stage_tables(sh, iv);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int4 w = __ldg(work + blockIdx.x);                  // {class, first tile, tiles, 0}
    const int4 cl = __ldg(pp.cls + w.x);
    unsigned long long ne = 0, nh = 0;
    for (int t = w.y + wid; t < w.y + w.z; t += kIdWarps) {
        const uint64_t rest = sp[(int64_t)t * 32 + lane];
        uint32_t am = 0, act = 0;
        for (int q = 0; q < cl.x; ++q) {
            const uint64_t m = __ldg(pp.mask + cl.y + q);
            const bool on = (rest & m) == 0 && lookup_index(iv, rest | m, sh.base_hi, sh.base_lo, sh.binom) >= 0;
            if (on) am |= 1u << q;
            if (__any_sync(kFull, on)) act |= 1u << q;
        }
        ne += __popc(am);
        for (uint32_t b = am; b; b &= b - 1u) nh += __popc(am & __ldg(pp.coup + cl.y + __ffs((int)b) - 1));
        int cnt = __popc(am);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(kFull, cnt, o);
        unsigned long long slot = 0, ent = 0;
        if (lane == 0) {
            slot = atomicAdd(tot + 2, 32ull * __popc(act));
            ent = atomicAdd(tot + 4, (unsigned long long)cnt);
            tile[t] = make_uint4(act, (uint32_t)slot, (uint32_t)ent, 0u);
        }
        slot = __shfl_sync(kFull, slot, 0) + lane;
        ent = __shfl_sync(kFull, ent, 0);
        for (uint32_t a = act; a; a &= a - 1u, slot += 32) {
            const int q = __ffs((int)a) - 1;
            uint32_t er = kNoEntry;
            const unsigned M = __ballot_sync(kFull, (am >> q) & 1u);
            if ((am >> q) & 1u) {
                const uint64_t m = __ldg(pp.mask + cl.y + q), s = rest | m;
                const int64_t j = lookup_index(iv, s, sh.base_hi, sh.base_lo, sh.binom);
                const int lo = __ffsll((long long)m) - 1, hi = 63 - __clzll((long long)m);
                const int v = above(s, lo), u = above(s, hi), k = v * (v - 1) / 2 + u;
                const unsigned long long e = ent + __popc(M & ((1u << lane) - 1u));
                if (j >= 0 && j < iv.n && k < kmax && slot < nslot && e < nent) {
                    er = (uint32_t)j | ((__popcll(rest & between(m)) & 1) ? 0x80000000u : 0u);
                    row_ent[(int64_t)k * iv.n + j] = (uint32_t)e;
                } else {
                    atomicAdd(tot + 3, 1ull);
                }
            }
            if (slot < nslot) ent_row[slot] = er;
            ent += __popc(M);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ne += __shfl_xor_sync(kFull, ne, o);
        nh += __shfl_xor_sync(kFull, nh, o);
    }
    if (lane == 0 && ne) {
        atomicAdd(tot, ne);
        atomicAdd(tot + 1, nh);
    }
}

template <typename R> __device__ __forceinline__ typename Cx<R>::T cx0() {
    typename Cx<R>::T v;
    v.x = 0;
    v.y = 0;
    return v;
}

// Four chains of FMAs per output; FP32 reads V two pairs at a time (16 bytes, as FP64 does one).
// A value is finite when its parts' high bits without their signs (top: the larger) are below kInf.
template <typename R> struct PairV;
template <> struct PairV<double> {
    static constexpr int kInf = 0x7ff00000;
    static __device__ __forceinline__ int top(double2 x) {
        return max(__double2hiint(x.x) & 0x7fffffff, __double2hiint(x.y) & 0x7fffffff);
    }
    static __device__ __forceinline__ double2 flip(double2 x, uint32_t sign) {
        return make_double2(__hiloint2double(__double2hiint(x.x) ^ (int)sign, __double2loint(x.x)),
                            __hiloint2double(__double2hiint(x.y) ^ (int)sign, __double2loint(x.y)));
    }
};
template <> struct PairV<float> {
    static constexpr int kInf = 0x7f800000;
    static __device__ __forceinline__ int top(float2 x) {
        return max(__float_as_int(x.x) & 0x7fffffff, __float_as_int(x.y) & 0x7fffffff);
    }
    static __device__ __forceinline__ float2 flip(float2 x, uint32_t sign) {
        return make_float2(__uint_as_float(__float_as_uint(x.x) ^ sign), __uint_as_float(__float_as_uint(x.y) ^ sign));
    }
};
// V[class][p][q] for the couplings of different pairs at parameter u: A + u B of their term slots
template <typename R>
__global__ void k_pair_values(const int32_t* __restrict__ vslot, int64_t nv, const typename Cx<R>::T* __restrict__ A,
                              const typename Cx<R>::T* __restrict__ B, R u, typename Cx<R>::T* __restrict__ V) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += (int64_t)gridDim.x * blockDim.x) {
        const int t = __ldg(vslot + i);
        typename Cx<R>::T a = cx0<R>();
        if (t >= 0) {
            a = A[t];
            if (B) {
                const typename Cx<R>::T b = B[t];
                a.x += u * b.x;
                a.y += u * b.y;
            }
        }
        V[i] = a;
    }
}

// Each row's diagonal, A and B parts in FP64: its one-body terms and its pairs with themselves, summed with
// their rounding errors (Knuth's two-sum), as the diagonal is most of a row.  With V[p][p] in the products instead, c64 maps were 1.1 to 3.2 times as far from 64 bits as over
// the hit records, which have the diagonal apart as well: 9.7e-8 against 3.6e-8 at 3x9 Ne = 9.
__global__ void k_pair_diag(PairPlanView pp, const uint64_t* __restrict__ basis, int64_t n,
                            const double2* __restrict__ A, const double2* __restrict__ B, double2* __restrict__ da,
                            double2* __restrict__ db) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double2 a = make_double2(0.0, 0.0), b = a, ea = a, eb = a;
        auto two = [](double& s, double& e, double v) {
            const double t = s + v, z = t - s;
            e += (s - (t - z)) + (v - z);
            s = t;
        };
        auto add = [&](int t) {
            if (t < 0) return;
            const double2 v = __ldg(A + t);
            two(a.x, ea.x, v.x);
            two(a.y, ea.y, v.y);
            if (B) {
                const double2 w = __ldg(B + t);
                two(b.x, eb.x, w.x);
                two(b.y, eb.y, w.y);
            }
        };
        for (uint64_t h = __ldg(basis + i); h; h &= h - 1ull) {
            const int lo = __ffsll((long long)h) - 1;
            add(__ldg(pp.d1 + lo));
            for (uint64_t g = h & (h - 1ull); g; g &= g - 1ull)
                add(__ldg(pp.d2 + lo * 64 + __ffsll((long long)g) - 1));
        }
        // (an infinite sum has no error to add)
        auto join = [](double s, double e) { return isfinite(e) ? s + e : s; };
        da[i] = make_double2(join(a.x, ea.x), join(a.y, ea.y));
        if (B) db[i] = make_double2(join(b.x, eb.x), join(b.y, eb.y));
    }
}

// row length of V in shared memory: even for FP32, whose loads take two values
template <typename R> __host__ __device__ constexpr int pair_ld(int pm) { return std::is_same<R, float>::value ? (pm + 1) / 2 * 2 : pm; }

// psi of the tiles of one work item: a lane per intermediate state, phi in registers (PM of them,
// the class's pairs padded with zeros), V broadcast from shared memory.  The loop over the outputs
// stays rolled: unrolled (13 x 13 products, ~20 KB of code that every warp runs once per tile) the
// kernel waited for instructions, 150 us instead of 84 on a 3x9 sector.
template <typename R, int PM>
__device__ __forceinline__ void pair_ids_body(const PairView& pv, int4 w, int P, const typename Cx<R>::T* __restrict__ Vs,
                                              const typename Cx<R>::T* __restrict__ x,
                                              typename Cx<R>::T* __restrict__ psi) {
    using C2 = typename Cx<R>::T;
    constexpr uint32_t kSign = 0x80000000u;
    constexpr int LD = pair_ld<R>(PM);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    for (int t = w.y + wid; t < w.y + w.z; t += kIdWarps) {
        const uint4 ti = __ldg(pv.tile + t);
        const uint32_t* er_p = pv.ent_row + ti.y + lane;
        C2 phi[PM];
        uint32_t er[PM], on = 0, sg = 0;
#pragma unroll
        for (int q = 0; q < PM; ++q) {
            er[q] = kNoEntry;
            if ((ti.x >> q) & 1u) {               // warp-uniform
                er[q] = ld_stream(er_p);
                er_p += 32;
            }
        }
#pragma unroll
        for (int q = 0; q < PM; ++q) {
            C2 v = cx0<R>();
            if (er[q] != kNoEntry) {
                v = __ldg(x + (er[q] & ~kSign));
                on |= 1u << q;
                sg |= (er[q] >> 31) << q;
            }
            phi[q] = PairV<R>::flip(v, er[q] & kSign);
        }
        C2* out = psi + ti.z;
#pragma unroll 1
        for (uint32_t a = ti.x; a; a &= a - 1u) {
            const int p = __ffs((int)a) - 1;
            const C2* v = Vs + p * LD;
            R ar = 0, ai = 0, br = 0, bi = 0;
            auto mac = [&](C2 c, int q) {
                ar += c.x * phi[q].x;
                ai += c.x * phi[q].y;
                br += c.y * phi[q].y;
                bi += c.y * phi[q].x;
            };
            if constexpr (std::is_same<R, float>::value) {
#pragma unroll
                for (int q = 0; q < PM; q += 2) {
                    const float4 c = *reinterpret_cast<const float4*>(v + q);
                    mac(make_float2(c.x, c.y), q);
                    if (q + 1 < PM) mac(make_float2(c.z, c.w), q + 1);
                }
            } else {
#pragma unroll
                for (int q = 0; q < PM; ++q) mac(v[q], q);
            }
            const unsigned M = __ballot_sync(kFull, (on >> p) & 1u);
            if ((on >> p) & 1u) {
                C2 o;
                o.x = ar - br;
                o.y = ai + bi;
                out[__popc(M & lt)] = PairV<R>::flip(o, (sg >> p) << 31);
            }
            out += __popc(M);
        }
    }
}

template <typename R, int PM>
__global__ void __launch_bounds__(kIdWarps * 32)
k_pair_ids(PairView pv, PairPlanView pp, const typename Cx<R>::T* __restrict__ V,
           const typename Cx<R>::T* __restrict__ x, typename Cx<R>::T* __restrict__ psi) {
    using C2 = typename Cx<R>::T;
    constexpr int PH = (PM + 1) / 2;              // classes of at most half the pairs (two components) pad to this
    __shared__ __align__(16) C2 Vs[PM * pair_ld<R>(PM)];
    const int4 w = __ldg(pv.work + blockIdx.x);
    const int4 cl = __ldg(pp.cls + w.x);
    const int P = cl.x, ld = pair_ld<R>(P <= PH ? PH : PM);
    for (int e = threadIdx.x; e < P * ld; e += kIdWarps * 32) {
        const int p = e / ld, q = e % ld;
        Vs[e] = q < P ? V[cl.z + p * P + q] : cx0<R>();
    }
    __syncthreads();
    if (P <= PH) pair_ids_body<R, PH>(pv, w, P, Vs, x, psi);
    else pair_ids_body<R, PM>(pv, w, P, Vs, x, psi);
}

// y[row] term by term, for a row whose sum is not finite.  psi takes couplings that the list lacks (V = 0)
// and pairs that a state lacks (phi = 0) along, which add nothing to finite values but spread an infinity
// or a NaN of x or V over the class; here it stays with the rows that the list connects to it.  Rare, so
// targets are searched in the sorted basis, and a test per row is all that the usual rows pay (48 registers
// instead of 32, before the rows' sums were FP64 throughout: 205 -> 200 us for c128 on 1.0M states, 16.6 ->
// 17.6 for c64 on 174k; held to 32: 224 and 20.4).  Tests in k_pair_ids cost 1 to 15% of the map, on its values, its products or once per tile.
template <typename R>
__device__ __noinline__ typename Cx<R>::T pair_row_apart(const PairPlanView& pp, const uint64_t* basis, int64_t n,
                                                         int64_t row, const typename Cx<R>::T* V, double2 d,
                                                         const typename Cx<R>::T* x) {
    using C2 = typename Cx<R>::T;
    const uint64_t s = basis[row];
    C2 acc = cx0<R>();
    bool diag = false;                                        // the row has a diagonal term
    auto add = [&](C2 c, int64_t j, bool neg) {
        const C2 v = x[j];
        const R pr = c.x * v.x - c.y * v.y, pi = c.x * v.y + c.y * v.x;
        acc.x += neg ? -pr : pr;
        acc.y += neg ? -pi : pi;
    };
#pragma unroll 1
    for (uint64_t h = s; h; h &= h - 1ull) {
        const int lo = __ffsll((long long)h) - 1;
        diag |= pp.d1[lo] >= 0;
#pragma unroll 1
        for (uint64_t g = h & (h - 1ull); g; g &= g - 1ull) {
            const int hi = __ffsll((long long)g) - 1, cs = pp.ptab[lo * 64 + hi];
            if (cs < 0) continue;
            diag |= pp.d2[lo * 64 + hi] >= 0;
            const int4 cl = pp.cls[cs >> 8];
            const int p = cs & 255;
            const uint64_t mp = (1ull << lo) | (1ull << hi), rest = s & ~mp;
#pragma unroll 1
            for (uint32_t m = pp.coup[cl.y + p]; m; m &= m - 1u) {
                const int q = __ffs((int)m) - 1;
                const uint64_t mq = pp.mask[cl.y + q], t = rest | mq;
                if (rest & mq) continue;
                int64_t b = 0, e = n;
                while (b < e) {
                    const int64_t c = (b + e) / 2;
                    if (basis[c] < t) b = c + 1;
                    else e = c;
                }
                if (b < n && basis[b] == t)
                    add(V[cl.z + p * cl.x + q], b, __popcll(rest & (between(mp) ^ between(mq))) & 1);
            }
        }
    }
    if (diag) {
        C2 c;
        c.x = (R)d.x;
        c.y = (R)d.y;
        add(c, row, false);
    }
    return acc;
}

// y[row] = sum of the psi of the row's pairs + diagonal x[row]: a lane per row, G warps share the pairs of 32
// rows (sums combined in a fixed order, in FP64 for FP32 values, too: 471 us against 445 in FP32 on two-
// component 4x6, where the error over the hit records' falls from 1.02 to 0.997).
template <typename R>
__global__ void __launch_bounds__(kPT, std::is_same<R, double>::value ? 4 : 5)    // no spills from here up
k_pair_rows(PairView pv, PairPlanView pp, const uint64_t* __restrict__ basis, const typename Cx<R>::T* __restrict__ V,
            const double2* __restrict__ da, const double2* __restrict__ db, double u,
            const typename Cx<R>::T* __restrict__ psi,
            const typename Cx<R>::T* __restrict__ x, typename Cx<R>::T* __restrict__ y, int G) {
    using C2 = typename Cx<R>::T;
    __shared__ double2 part[kPT];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int g = wid % G;
    const int64_t row = ((int64_t)blockIdx.x * (kPT / 32 / G) + wid / G) * 32 + lane;
    double2 acc = make_double2(0.0, 0.0);
    if (row < pv.n) {
        const uint32_t* re = pv.row_ent + row;
        // pairs in flight: 12 FP32 values take the registers of 6 FP64 ones.  c64 with 6 / 12, in us: 99.2 /
        // 97.2 on 247k states, 68.3 / 66.8 on 131k, 64.4 / 62.3 on 276k (two components), 457 / 448 on 1.0M
        constexpr int U = std::is_same<R, double>::value ? 6 : 12;
        for (int k = g; k < pv.kmax; k += U * G) {
            uint32_t e[U];
            C2 v[U];
#pragma unroll
            for (int i = 0; i < U; ++i) e[i] = k + i * G < pv.kmax ? ld_stream(re + (int64_t)(k + i * G) * pv.n) : kNoEntry;
#pragma unroll
            for (int i = 0; i < U; ++i) v[i] = e[i] != kNoEntry ? __ldg(psi + e[i]) : cx0<R>();
#pragma unroll
            for (int j = 0; j < U; j += 6) {
#pragma unroll
                for (int i = j; i < j + 3; ++i) { v[i].x += v[i + 3].x; v[i].y += v[i + 3].y; }
                acc.x += v[j].x + (v[j + 1].x + v[j + 2].x);
                acc.y += v[j].y + (v[j + 1].y + v[j + 2].y);
            }
        }
    }
    double2 d = make_double2(0.0, 0.0);
    C2 xv = cx0<R>();
    if (g == 0 && row < pv.n) {
        d = __ldg(da + row);
        xv = __ldg(x + row);
        if (db) {
            const double2 b = __ldg(db + row);
            d.x += u * b.x;
            d.y += u * b.y;
        }
    }
    if (G > 1) {
        part[threadIdx.x] = acc;
        __syncthreads();
        if (g == 0) {
            for (int i = 1; i < G; ++i) {
                const double2 v = part[threadIdx.x + 32 * i];
                acc.x += v.x;
                acc.y += v.y;
            }
        }
    }
    if (g == 0 && row < pv.n) {
        C2 o;                                     // the diagonal is most of y: joined and rounded once
        o.x = (R)fma(d.x, (double)xv.x, fma(-d.y, (double)xv.y, acc.x));
        o.y = (R)fma(d.x, (double)xv.y, fma(d.y, (double)xv.x, acc.y));
        if (PairV<R>::top(o) >= PairV<R>::kInf) o = pair_row_apart<R>(pp, basis, pv.n, row, V, d, x);
        y[row] = o;
    }
}

int pair_sms() {
    static const int s = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 148;
    }();
    return s;
}

template <typename T> void upload(DevBuf<T>& dst, const std::vector<T>& src, cudaStream_t st) {
    dst.resize(std::max<size_t>(src.size(), 1));
    if (!src.empty()) MOMED_CUDA_TRY(cudaMemcpyAsync(dst.p, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice, st));
}

}  // namespace

PairPlanView PairPlan::view() const {
    PairPlanView v{};
    v.nclass = nclass;
    v.cls = cls.p;
    v.mask = mask.p;
    v.coup = coup.p;
    v.ptab = ptab.p;
    v.d1 = d1.p;
    v.d2 = d2.p;
    return v;
}

PairView PairMap::view() const {
    PairView v{};
    v.n = n;
    v.kmax = kmax;
    v.tile = tile.p;
    v.ent_row = ent_row.p;
    v.row_ent = row_ent.p;
    v.work = work.p;
    return v;
}

// The pair classes of the working operator (once per uploaded term list).  The pair form takes
// operators whose off-diagonal terms are all two-body, with classes of at most 32 pairs and no term
// listed twice.
bool pair_plan(momed_handle* h) {
    PairPlan& pl = h->pplan;
    if (pl.state >= 0) return pl.state == 1;
    pl.state = 0;
    const std::vector<uint64_t>&tin = h->op.h_in, &tout = h->op.h_out;
    const int64_t nt = (int64_t)tin.size();
    std::vector<uint64_t> pairs;
    std::vector<int32_t> d1(64, -1);
    for (int64_t t = 0; t < nt; ++t) {
        if (t > 0 && tin[t] == tin[t - 1] && tout[t] == tout[t - 1]) return false;   // listed twice (sorted by out, in)
        const int b = __builtin_popcountll(tout[t]);
        if (b == 1) {
            if (tin[t] != tout[t]) return false;
            d1[__builtin_ctzll(tout[t])] = (int32_t)t;
        } else if (b == 2) {
            pairs.push_back(tin[t]);
            pairs.push_back(tout[t]);
        } else {
            return false;
        }
    }
    std::sort(pairs.begin(), pairs.end());
    pairs.erase(std::unique(pairs.begin(), pairs.end()), pairs.end());
    const int np = (int)pairs.size();
    if (np == 0) return false;
    auto at = [&](uint64_t m) { return (int)(std::lower_bound(pairs.begin(), pairs.end(), m) - pairs.begin()); };
    std::vector<int> up(np);
    std::iota(up.begin(), up.end(), 0);
    auto root = [&](int i) {
        while (up[i] != i) i = up[i] = up[up[i]];
        return i;
    };
    for (int64_t t = 0; t < nt; ++t)
        if (__builtin_popcountll(tout[t]) == 2) {
            const int a = root(at(tout[t])), b = root(at(tin[t]));
            if (a != b) up[std::max(a, b)] = std::min(a, b);
        }
    std::vector<int> cls_of(np, -1), slot_of(np, 0), P;
    for (int i = 0; i < np; ++i) {
        const int r = root(i);
        if (cls_of[r] < 0) {
            cls_of[r] = (int)P.size();
            P.push_back(0);
        }
        cls_of[i] = cls_of[r];
        slot_of[i] = P[cls_of[i]]++;
        if (P[cls_of[i]] > kMaxClassPairs) return false;
    }
    const int nc = (int)P.size();
    if (nc > kMaxClasses) return false;
    std::vector<int4> cls(nc);
    int64_t moff = 0, voff = 0;
    int pmax = 0;
    for (int c = 0; c < nc; ++c) {
        cls[c] = make_int4(P[c], (int)moff, (int)voff, 0);
        moff += P[c];
        voff += (int64_t)P[c] * P[c];
        pmax = std::max(pmax, P[c]);
    }
    std::vector<uint64_t> mask(np);
    std::vector<uint32_t> coup(np, 0u);
    std::vector<int32_t> ptab(64 * 64, -1), d2(64 * 64, -1), vslot(voff, -1);
    for (int i = 0; i < np; ++i) {
        mask[cls[cls_of[i]].y + slot_of[i]] = pairs[i];
        const int lo = __builtin_ctzll(pairs[i]), hi = 63 - __builtin_clzll(pairs[i]);
        ptab[lo * 64 + hi] = cls_of[i] << 8 | slot_of[i];
    }
    int64_t ncoup = 0;
    for (int64_t t = 0; t < nt; ++t)
        if (__builtin_popcountll(tout[t]) == 2) {
            const int o = at(tout[t]), i = at(tin[t]);
            const int4 c = cls[cls_of[o]];
            if (o == i) {
                d2[__builtin_ctzll(pairs[o]) * 64 + 63 - __builtin_clzll(pairs[o])] = (int32_t)t;
            } else {
                vslot[c.z + slot_of[o] * c.x + slot_of[i]] = (int32_t)t;
                coup[c.y + slot_of[o]] |= 1u << slot_of[i];
                ++ncoup;
            }
        }
    cudaStream_t st = h->stream;
    upload(pl.cls, cls, st);
    upload(pl.mask, mask, st);
    upload(pl.coup, coup, st);
    upload(pl.ptab, ptab, st);
    upload(pl.vslot, vslot, st);
    upload(pl.d1, d1, st);
    upload(pl.d2, d2, st);
    MOMED_CUDA_TRY(cudaStreamSynchronize(st));
    pl.P = P;
    pl.nclass = nc;
    pl.pmax = pmax;
    pl.nv = voff;
    pl.density = voff > np ? (double)ncoup / (double)(voff - np) : 0.0;
    pl.state = 1;
    return true;
}

// most pairs a basis state can have, from the largest particle number in the basis
static int64_t pairs_per_row(const momed_handle* h) {
    const int64_t ne = h->basis_pop_max;
    return ne * (ne - 1) / 2;
}

// Device memory of the tables, the FP64 workspace and the build, by the basis alone: row_ent and psi per
// (row, pair), ent_row per slot (twice as many as entries: half of a class's pairs free in a state; 1.9 at
// 3x9 Ne = 9, 2.2 at 5x5 Ne = 10), the tables and workspace of the states, and the rows' diagonals.  The build counts slots and
// states before it allocates, and asks again where they take more.
int64_t pair_bytes(const momed_handle* h) {
    const int64_t e = h->n * pairs_per_row(h);
    return e * (4 + 16) + 2 * e * 4 + e * 8 / 3 + h->n * 32;
}

// MOMED_PAIRMAP=0: never, =1: whatever the size and density
static int pair_policy() {
    const char* e = std::getenv("MOMED_PAIRMAP");
    return e && (e[0] == '0' || e[0] == '1') ? e[0] - '0' : -1;
}

// Below 2^20 entries the two launches of a product lose what the gathers save: on the B200, FP64 /
// FP32, against the hit records, 30.6k states x 28 pairs (858k entries) 26.7 / 23.1 us against 28-29
// / 21.2, 7.1k x 15 (106k) 17.5 / 16.9 against 12.1 / 10.6, but 43k x 28 (1.2M) 28.4 / 25.3 against
// 40.3 / 28.9.
constexpr int64_t kMinEntries = 1 << 20;
// Hits an entry has to stand for: the records visit them one by one, the pair form takes P products
// instead, so a nearly half-filled lattice (few free pairs per state) gains nothing.  3.4 hits per
// entry (4x6 Ne = 11) ran 109 us against 98, 4.4 (5x5 Ne = 10) 98 against 126, 4.7 (3x9 Ne = 11)
// 437 against 546, 6.0 (3x9 Ne = 9) 108 against 180, 6.5 (4x7 Ne = 9) 147 against 261.
constexpr double kMinHitsPerEntry = 4.0;

bool pair_possible(momed_handle* h) {
    const int64_t k = pairs_per_row(h);
    if (h->hcache.pair.declined || pair_policy() == 0) return false;
    if (pair_policy() != 1 && h->n * k < kMinEntries) return false;
    if (h->n <= 0 || h->n >= (int64_t)0x7fffffff || k < 1 || k > 2016) return false;
    if (h->n * k >= (int64_t)kNoEntry) return false;      // entries are 32-bit, and so is a row block's item count
    return pair_plan(h);
}

// the rows' diagonals from the term amplitudes
static void pair_diag(momed_handle* h) {
    PairMap& pm = h->hcache.pair;
    const OpView ov = h->op.view();
    pm.da.resize(pm.n);
    if (ov.t_ampb) pm.db.resize(pm.n);
    k_pair_diag<<<(unsigned)std::min<int64_t>((pm.n + 255) / 256, 1184), 256, 0, h->stream>>>(
        h->pplan.view(), h->basis.p, pm.n, ov.t_amp, ov.t_ampb, pm.da.p, pm.db.p);
    MOMED_CUDA_TRY(cudaGetLastError());
    note_launches(1);
    pm.ok_diag = true;
}

// Builds the tables (the caller has the index; lookups compare keys, so no validation of the
// operator is needed).  Returns false, with nothing built, where the states have too few free pairs or
// the tables do not fit after all.
bool build_pair_map(momed_handle* h, double share) {
    PairMap& pm = h->hcache.pair;
    pm.release();
    const PairPlan& pl = h->pplan;
    cudaStream_t st = h->stream;
    IndexView iv = index_view(h);
    if (iv.mode == INDEX_RANKED) iv.mode = INDEX_CHECKED;
    const PairPlanView pp = pl.view();
    const int64_t n = h->n;
    const int kmax = (int)pairs_per_row(h);
    const int64_t nent = n * kmax;
    // row blocks: enough to fill the device, few enough for the class scan
    const int64_t rpb = std::max<int64_t>(32, (n + 1183) / 1184);
    const int nblk = (int)((n + rpb - 1) / rpb);
    DevBuf<uint8_t> own;
    DevBuf<int32_t> counts, total, cbase;
    own.resize(nent);
    counts.resize((size_t)nblk * pl.nclass);
    total.resize(pl.nclass);
    cbase.resize(pl.nclass);
    DevBuf<unsigned long long> tot;
    tot.resize(5);
    MOMED_CUDA_TRY(cudaMemsetAsync(tot.p, 0, 5 * sizeof(unsigned long long), st));
    const size_t hs = (size_t)pl.nclass * sizeof(int);
    k_pair_own<<<nblk, kPT, hs, st>>>(iv, pp, kmax, rpb, own.p, counts.p);
    k_pair_scan<<<(pl.nclass + 7) / 8, 256, 0, st>>>(counts.p, nblk, pl.nclass, total.p);
    MOMED_CUDA_TRY(cudaGetLastError());
    std::vector<int32_t> tc(pl.nclass), cb(pl.nclass);
    MOMED_CUDA_TRY(cudaMemcpyAsync(tc.data(), total.p, tc.size() * 4, cudaMemcpyDeviceToHost, st));
    MOMED_CUDA_TRY(cudaStreamSynchronize(st));
    int64_t tiles = 0, slots = 0;              // slots: every tile with every pair of its class
    for (int c = 0; c < pl.nclass; ++c) {
        cb[c] = (int32_t)(tiles * 32);
        tiles += (tc[c] + 31) / 32;
        slots += (int64_t)(tc[c] + 31) / 32 * 32 * pl.P[c];
    }
    const int64_t pad = tiles * 32;
    const int64_t ids = std::accumulate(tc.begin(), tc.end(), (int64_t)0);
    if (pair_policy() != 1 && ((double)nent / (double)std::max<int64_t>(ids, 1) - 1.0) * pl.density < kMinHitsPerEntry) {
        pm.declined = true;
        return false;
    }
    const int64_t need = nent * (4 + 16 + 1) + slots * 4 + tiles * 16 + pad * 8 + n * 32;
    if (need > pair_bytes(h) && !(share > 0.0 && fits_free(need, share))) {
        pm.declined = true;
        return false;
    }
    std::vector<int2> win;                     // sorting windows, class by class
    for (int c = 0; c < pl.nclass; ++c)
        for (int i = 0; i < tc[c]; i += kSortIds) win.push_back(make_int2(cb[c] + i, std::min(kSortIds, tc[c] - i)));
    MOMED_REQUIRE(pad < (int64_t)0x7fffffff && slots < (int64_t)kNoEntry, MOMED_ENOMEM,
                  "pair map: too many intermediate states");
    // work items: runs of tiles of one class, so that V is staged once per block; at least one
    // tile per warp, up to 16 on large sectors (about three waves of blocks)
    const int64_t per = std::min<int64_t>(16 * kIdWarps, std::max<int64_t>(kIdWarps, tiles / (pair_sms() * 12) / kIdWarps * kIdWarps));
    std::vector<int4> work;
    for (int c = 0; c < pl.nclass; ++c) {
        const int t0 = cb[c] / 32, nt = (tc[c] + 31) / 32;
        for (int t = 0; t < nt; t += (int)per) work.push_back(make_int4(c, t0 + t, (int)std::min<int64_t>(per, nt - t), 0));
    }
    pm.nwork = (int)work.size();
    upload(pm.work, work, st);
    MOMED_CUDA_TRY(cudaMemcpyAsync(cbase.p, cb.data(), cb.size() * 4, cudaMemcpyHostToDevice, st));
    DevBuf<uint64_t> sp;
    sp.resize(std::max<int64_t>(pad, 1));
    pm.tile.resize(std::max<int64_t>(tiles, 1));
    pm.ent_row.resize(std::max<int64_t>(slots, 1));
    pm.row_ent.resize(std::max<int64_t>(nent, 1));
    MOMED_CUDA_TRY(cudaMemsetAsync(sp.p, 0xFF, pad * 8, st));
    MOMED_CUDA_TRY(cudaMemsetAsync(pm.row_ent.p, 0xFF, nent * 4, st));
    DevBuf<int2> wind;
    upload(wind, win, st);
    k_pair_assign<<<nblk, kPT, hs, st>>>(iv, pp, kmax, rpb, own.p, counts.p, cbase.p, sp.p);
    if (!win.empty()) k_pair_sort<<<(unsigned)win.size(), 1024, 0, st>>>(wind.p, sp.p);
    if (pm.nwork > 0)
        k_pair_fill<<<pm.nwork, kIdWarps * 32, 0, st>>>(iv, pp, pm.work.p, sp.p, pm.tile.p, pm.ent_row.p,
                                                        pm.row_ent.p, kmax, (unsigned long long)slots,
                                                        (unsigned long long)nent, tot.p);
    MOMED_CUDA_TRY(cudaGetLastError());
    note_launches(pm.nwork > 0 ? 5 : 3);
    unsigned long long th[5] = {0, 0, 0, 0, 0};
    MOMED_CUDA_TRY(cudaMemcpyAsync(th, tot.p, sizeof(th), cudaMemcpyDeviceToHost, st));
    MOMED_CUDA_TRY(cudaStreamSynchronize(st));   // also keeps the uploaded vectors alive until their copies ran
    if (th[3] != 0 || th[0] != th[4] || th[0] > (unsigned long long)nent || th[2] > (unsigned long long)slots) {
        pm.release();
        throw Error{MOMED_EINVAL, "pair map: table passes disagree"};
    }
    pm.kmax = kmax;
    pm.entries = (int64_t)th[0];
    // here, so that the first product does not wait for them
    pm.psi.resize(std::max<int64_t>(pm.entries, 1));
    pm.n = n;
    pair_diag(h);
    pm.hits = (int64_t)th[1];
    pm.bytes = (int64_t)(pm.work.bytes() + pm.tile.bytes() + pm.ent_row.bytes() + pm.row_ent.bytes() + pm.psi.bytes() +
                         pm.da.bytes() + pm.db.bytes());
    pm.built = true;
    return true;
}

namespace {

template <typename R> struct PairSlot;
template <> struct PairSlot<double> {
    static DevBuf<double2>& v(PairPlan& p) { return p.v64; }
    static double& u(PairMap& m) { return m.u64; }
    static bool& ok(PairMap& m) { return m.ok64; }
    static const double2* a(const OpView& o) { return o.t_amp; }
    static const double2* b(const OpView& o) { return o.t_ampb; }
};
template <> struct PairSlot<float> {
    static DevBuf<float2>& v(PairPlan& p) { return p.v32; }
    static double& u(PairMap& m) { return m.u32; }
    static bool& ok(PairMap& m) { return m.ok32; }
    static const float2* a(const OpView& o) { return o.t_amp32; }
    static const float2* b(const OpView& o) { return o.t_ampb32; }
};

template <typename R, int PM>
void ids_launch(const PairMap& pm, const PairPlan& pl, const typename Cx<R>::T* V, const typename Cx<R>::T* x,
                typename Cx<R>::T* psi, cudaStream_t st) {
    k_pair_ids<R, PM><<<pm.nwork, kIdWarps * 32, 0, st>>>(pm.view(), pl.view(), V, x, psi);
}

template <typename R>
void pair_apply(momed_handle* h, const typename Cx<R>::T* x, typename Cx<R>::T* y, double u, cudaStream_t st) {
    using S = PairSlot<R>;
    using C2 = typename Cx<R>::T;
    PairPlan& pl = h->pplan;
    PairMap& pm = h->hcache.pair;
    MOMED_REQUIRE(pm.built && pm.n == h->n, MOMED_ESTATE, "pair map: not built");
    if (pm.n <= 0) return;
    const OpView ov = h->op.view();
    auto& V = S::v(pl);
    C2* psi = reinterpret_cast<C2*>(pm.psi.p);
    if (!S::ok(pm) || (ov.t_ampb && S::u(pm) != u)) {         // formed again for another u or new amplitudes
        V.resize(std::max<int64_t>(pl.nv, 1));
        k_pair_values<R><<<(unsigned)std::min<int64_t>((pl.nv + 255) / 256, 1184), 256, 0, st>>>(
            pl.vslot.p, pl.nv, S::a(ov), S::b(ov), (R)u, V.p);
        MOMED_CUDA_TRY(cudaGetLastError());
        note_launches(1);
        if (!pm.ok_diag) pair_diag(h);                        // new amplitudes without a rebuild
        S::u(pm) = u;
        S::ok(pm) = true;
    }
    if (pm.nwork > 0) {
        // instantiated pair counts: every even one to 16 and of the odd ones 13 and 15 (meshes of 26, 27
        // and 30, 31 orbitals, 3x9 and 3x10 among them), then steps of 4; a class pads to the next (11 pairs,
        // of 22 and 23 orbitals, to 12)
        switch (pl.pmax <= 4 ? 4 : pl.pmax <= 16 ? (pl.pmax == 13 || pl.pmax == 15 ? pl.pmax : (pl.pmax + 1) / 2 * 2)
                                                 : (pl.pmax + 3) / 4 * 4) {
            case 4: ids_launch<R, 4>(pm, pl, V.p, x, psi, st); break;
            case 6: ids_launch<R, 6>(pm, pl, V.p, x, psi, st); break;
            case 8: ids_launch<R, 8>(pm, pl, V.p, x, psi, st); break;
            case 10: ids_launch<R, 10>(pm, pl, V.p, x, psi, st); break;
            case 12: ids_launch<R, 12>(pm, pl, V.p, x, psi, st); break;
            case 13: ids_launch<R, 13>(pm, pl, V.p, x, psi, st); break;
            case 14: ids_launch<R, 14>(pm, pl, V.p, x, psi, st); break;
            case 15: ids_launch<R, 15>(pm, pl, V.p, x, psi, st); break;
            case 16: ids_launch<R, 16>(pm, pl, V.p, x, psi, st); break;
            case 20: ids_launch<R, 20>(pm, pl, V.p, x, psi, st); break;
            case 24: ids_launch<R, 24>(pm, pl, V.p, x, psi, st); break;
            case 28: ids_launch<R, 28>(pm, pl, V.p, x, psi, st); break;
            default: ids_launch<R, 32>(pm, pl, V.p, x, psi, st); break;
        }
        MOMED_CUDA_TRY(cudaGetLastError());
        note_launches(1);
    }
    // Warps per 32 rows: enough of them to cover the gathers' latency on small sectors, 16 an SM; more
    // only share the row's sums.  A map with 1 / 2 / 4 of them, in us: c128 30.4 / 28.4 / 30.2 on 43k
    // states (1.4k warps of rows), 98.5 / 100.4 / 104 on 131k, 107.9 / 105.9 / 109.9 on 174k, 146.4 / 148.7 /
    // 152.8 on 247k; c64 with 1 / 2 24.3 / 24.4, 66.8 / 68.9, 69.3 / 71.1, 97.2 / 99.2.
    // (64 an SM, for a kernel of 32 registers, cost this one up to 17%: 115.1 on 131k states, c128.)
    const int64_t rw = (pm.n + 31) / 32, want = (int64_t)pair_sms() * 16;
    int G = 1;
    while (G < 8 && rw * G < want) G *= 2;
    const int per = kPT / 32 / G;
    k_pair_rows<R><<<(unsigned)((rw + per - 1) / per), kPT, 0, st>>>(pm.view(), pl.view(), h->basis.p, V.p, pm.da.p, ov.t_ampb ? pm.db.p : nullptr,
                                                                     u, psi, x, y, G);
    MOMED_CUDA_TRY(cudaGetLastError());
    note_launches(1);
}

}  // namespace

void launch_pair_c128(momed_handle* h, const double2* x, double2* y, double u, cudaStream_t st) {
    pair_apply<double>(h, x, y, u, st);
}
void launch_pair_c64(momed_handle* h, const float2* x, float2* y, double u, cudaStream_t st) {
    pair_apply<float>(h, x, y, u, st);
}

}  // namespace momed
