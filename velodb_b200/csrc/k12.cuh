// Union-sort operators on 12-byte rows (RowK12: u64 key k, u32 payload p): the
// forward fill over the sorted rows and the row layouts of the oblivious gather
// and the PK-FK join of the plain path (ops.cu).
//
// Gather row: k = (row id | table row count clamp) << 33 | request << 32
//                 | high half of x, p = low half of x; x = the table's value, or
//             the number of the request.  After the fill a request becomes
//             k = number << 32 | high half of the value, p = low half of it, and
//             a table row the largest row, so that a sort brings the requests
//             back in order.
// Join row:   k = order-preserving key, p = tag (1 probe) << 31 | valid << 30
//             | row id.  After the fill a joined probe row becomes the word
//             build row << 30 | probe row, any other row ~0.
#pragma once

#include "union.cuh"

namespace velo {

constexpr int K12_TS = 2048, K12_THREADS = 256, K12_RPT = K12_TS / K12_THREADS;
// slot of tile row i: one pad word after every 8 rows, so that the 8 rows of
// neighbouring threads fall in different banks
__device__ __forceinline__ int k12_slot(int i) { return i + (i >> 3); }
constexpr int K12_TS_PAD = K12_TS + K12_TS / K12_RPT;

constexpr uint32_t OG_NONE = 0x7FFFFFFFu; // row id of a request past the table

struct GatherK12 {
    struct Out {
        uint64_t* k;
        uint32_t* p;
    };
    __device__ __forceinline__ static FillCarry src(uint64_t k, uint32_t p)
    {
        return FillCarry { 0, (k << 32) | p, ((k >> 32) & 1ull) == 0 ? 1u : 0u, 1u };
    }
    __device__ __forceinline__ static bool dup(uint64_t, uint32_t, const FillCarry&) { return false; }
    // every row id below the table size has its table row, the last one before
    // the requests for it
    __device__ __forceinline__ static void apply(uint64_t& k, uint32_t& p, const FillCarry& last)
    {
        const bool req = ((k >> 32) & 1ull) != 0;
        const uint64_t val = (uint32_t)(k >> 33) == OG_NONE ? 0ull : last.val;
        k = req ? ((uint64_t)p << 32) | (val >> 32) : ~0ull;
        p = req ? (uint32_t)val : ~0u;
    }
    __device__ __forceinline__ static void store(const Out& o, size_t g, uint64_t k, uint32_t p)
    {
        o.k[g] = k;
        o.p[g] = p;
    }
};

constexpr uint32_t OJ12_TAG = 1u << 31, OJ12_VALID = 1u << 30, OJ12_ROWID = OJ12_VALID - 1u;

struct JoinK12 {
    struct Out {
        uint64_t* w;
    };
    __device__ __forceinline__ static bool is_pad(uint64_t k, uint32_t p) { return k == ~0ull && p == ~0u; }
    __device__ __forceinline__ static FillCarry src(uint64_t k, uint32_t p)
    {
        return FillCarry { k, p & OJ12_ROWID, (p & OJ12_TAG) ? 0u : 1u, (p & OJ12_VALID) ? 1u : 0u };
    }
    // a build row whose key equals the preceding build row's key
    __device__ __forceinline__ static bool dup(uint64_t k, uint32_t p, const FillCarry& last)
    {
        return ((p & OJ12_TAG) == 0) & (last.has != 0) & (last.key == k);
    }
    __device__ __forceinline__ static void apply(uint64_t& k, uint32_t& p, const FillCarry& last)
    {
        const bool joined = ((p & (OJ12_TAG | OJ12_VALID)) == (OJ12_TAG | OJ12_VALID)) & !is_pad(k, p) & (last.has != 0)
            & (last.valid != 0) & (last.key == k);
        k = joined ? (last.val << 30) | (p & OJ12_ROWID) : ~0ull;
    }
    __device__ __forceinline__ static void store(const Out& o, size_t g, uint64_t k, uint32_t) { o.w[g] = k; }
};

// the last source row of each tile of the rows [0, n)
template <class F>
__global__ void __launch_bounds__(K12_THREADS) k_k12_sum(const uint64_t* k, const uint32_t* p, size_t n,
                                                         FillCarry* tile_last)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_k12_sum"));
    __shared__ FillCarry sm[K12_THREADS / 32];
    __shared__ int idx[K12_THREADS / 32];
    const size_t base = (size_t)blockIdx.x * K12_TS;
    FillCarry c { 0, 0, 0, 0 };
    int last = -1;
#pragma unroll
    for (int r = 0; r < K12_RPT; r++) {
        const int i = r * K12_THREADS + (int)threadIdx.x;
        const size_t g = base + i;
        if (g < n) {
            VELO_TRACE_AT(TS_FILL, k + g);
            const FillCarry d = F::src(k[g], p[g]);
            c = fill_combine(c, d);
            last = d.has ? i : last;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const FillCarry oc = fill_shfl(c, off, false);
        const int oi = __shfl_xor_sync(0xFFFFFFFFu, last, off);
        const bool take = oi > last;
        c = take ? oc : c;
        last = take ? oi : last;
    }
    if ((threadIdx.x & 31) == 0) {
        sm[threadIdx.x >> 5] = c;
        idx[threadIdx.x >> 5] = last;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < K12_THREADS / 32; w++) {
            const bool take = idx[w] > last;
            c = take ? sm[w] : c;
            last = take ? idx[w] : last;
        }
        VELO_TRACE_AT(TS_FILL, tile_last + blockIdx.x);
        tile_last[blockIdx.x] = c;
    }
}

// fill of the rows [0, n): loads and stores pass through shared memory, so
// that a thread owns 8 consecutive rows and the global accesses stay coalesced
template <class F>
__global__ void __launch_bounds__(K12_THREADS) k_k12_apply(const uint64_t* k, const uint32_t* p, size_t n,
                                                           const FillCarry* carry, typename F::Out out,
                                                           unsigned long long* d_stat)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_k12_apply"));
    __shared__ uint64_t sk[K12_TS_PAD];
    __shared__ uint32_t sp[K12_TS_PAD];
    __shared__ FillCarry wsm[33];
    __shared__ uint32_t tmp[33];
    const size_t base = (size_t)blockIdx.x * K12_TS;
#pragma unroll
    for (int r = 0; r < K12_RPT; r++) {
        const int i = r * K12_THREADS + (int)threadIdx.x;
        const size_t g = base + i;
        if (g < n) {
            VELO_TRACE_AT(TS_FILL, k + g);
            sk[k12_slot(i)] = k[g];
            sp[k12_slot(i)] = p[g];
        }
    }
    __syncthreads();
    const int s0 = (int)threadIdx.x * (K12_RPT + 1);
    const size_t g0 = base + (size_t)threadIdx.x * K12_RPT;
    uint64_t a[K12_RPT];
    uint32_t b[K12_RPT];
    FillCarry mine { 0, 0, 0, 0 };
#pragma unroll
    for (int r = 0; r < K12_RPT; r++) {
        a[r] = sk[s0 + r];
        b[r] = sp[s0 + r];
        if (g0 + r < n)
            mine = fill_combine(mine, F::src(a[r], b[r]));
    }
    FillCarry run = fill_combine(carry[blockIdx.x], block_fill_scan_excl(mine, wsm));
    uint32_t stat = 0;
#pragma unroll
    for (int r = 0; r < K12_RPT; r++) {
        if (g0 + r < n) {
            stat += F::dup(a[r], b[r], run) ? 1u : 0u;
            run = fill_combine(run, F::src(a[r], b[r]));
            F::apply(a[r], b[r], run);
        }
        sk[s0 + r] = a[r];
        sp[s0 + r] = b[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < K12_RPT; r++) {
        const int i = r * K12_THREADS + (int)threadIdx.x;
        const size_t g = base + i;
        if (g < n) {
            VELO_TRACE_AT(TS_FILL, k + g);
            F::store(out, g, sk[k12_slot(i)], sp[k12_slot(i)]);
        }
    }
    // one counter update per CTA at a fixed address
    uint32_t total;
    block_exclusive_scan(stat, tmp, &total);
    if (threadIdx.x == 0 && d_stat)
        atomicAdd(d_stat, (unsigned long long)total);
}

template <class F>
static velo_status run_fill_k12(const uint64_t* k, const uint32_t* p, size_t n, const typename F::Out& out,
                                FillCarry* tl, FillCarry* carry, unsigned long long* d_stat, cudaStream_t st)
{
    static_assert(K12_TS == FL_TS, "the tile carries of union_layout");
    const int nt = (int)((n + K12_TS - 1) / K12_TS);
    k_k12_sum<F><<<nt, K12_THREADS, 0, st>>>(k, p, n, tl);
    k_fill_scan<<<1, 1024, 0, st>>>(tl, nt, carry);
    k_k12_apply<F><<<nt, K12_THREADS, 0, st>>>(k, p, n, carry, out, d_stat);
    VELO_CUDA_TRY(cudaGetLastError(), "fill launch");
    return VELO_OK;
}

} // namespace velo
