// Oblivious filter + group-by over a lineitem-shaped fact table.
//
// The public bound on the groups (at most 16) lets the query run without
// moving the table's rows: the group keys are found first, then one pass adds
// every row into the slot of its key with masks.  All on the device, one
// stream, no host round trip:
//   1. keys     predicate (conjunctive ranges, the pushed-down WHERE of
//               src/operator/seq_scan_operator.cpp:38-45 evaluated on the GPU);
//               each row becomes a 16-bit key flag1 << 8 | flag2, or 0xFFFF if
//               it fails the filter; rows that pass with the real key 0xFFFF
//               are counted.  Row i and row i + h, h = ceil(n / 2), share a
//               32-bit word (RowU2).
//   2. sort     bitonic network on the words: both 16-bit lanes sorted at
//               once; then the smaller and the larger of (low lane i, high lane
//               N - 1 - i) and one more merge, which leaves the lower half of
//               all keys sorted in the low lane and the upper half in the high
//               lane
//   3. groups   rows whose key differs from the one before are the groups, in
//               key order; a prefix count ranks them and each of the first
//               group_bound becomes a slot
//   4. sums     every row is added to every slot with a mask (exact int64)
// It replaces FilterCompactionOperator's scatter/gather
// (src/operator/filter_compaction_operator.cpp:65-184) and the sorted
// segmented sums of obliviator/operator_2/enclave/
// scalable_oblivious_join.c:221-262: the same groups, counts and sums.  The
// order of the passes and every address depend on n and group_bound alone.
//
// Why: sorting 16-byte records of next_pow2(n) rows took 1.74 ms of a 2.17 ms
// call at 6,001,215 rows (ORCompact 0.31 ms, aggregation 0.29 ms).  The keys
// are an eighth of the bytes, an exchange of two keys is four instructions
// instead of two exchanges of about 19, and the rows' 26 bytes are read once
// here.  6,001,215 rows: 2,166 -> 542 us (keys 23, sort 386, groups 39, sums
// 104).
#include "net_host.cuh"
#include "groupby.cuh"

namespace velo {

// 16,384-row tiles of 512 threads x 32 rows: 64 KB of shared memory, and the
// 14 levels of a merge in three windows
constexpr int LK_LOG_NT = 9, LK_LOG_E = 5, LK_LT = LK_LOG_NT + LK_LOG_E, LK_LMAX = 9;
constexpr int LK_THREADS = 256;
constexpr int LK_ROWS = 1024; // key words of a CTA's first grid-stride step
constexpr int LK_TS = 4096;   // key words of a tile of the group search
constexpr uint32_t LK_NONE = 0xFFFFu;
constexpr unsigned LK_MAX_BLOCKS = 148 * 8;

// the words the later steps share (in the 256 bytes of LiScratch::d_rows)
struct LkMeta {
    uint64_t rows;   // rows passing the filter
    uint64_t groups; // distinct keys among them
    uint32_t slot[SEG_MAX_G]; // key + 1 of group j, 0 past the last group
};
static_assert(sizeof(LkMeta) <= 256, "fits the 256-byte aligned area of d_rows");

__device__ __forceinline__ bool li_pass(const LiCols& c, const velo_lineitem_pred& p, size_t g)
{
    const int32_t q = c.qty[g], d = c.disc[g], s = c.ship[g];
    return (s >= p.ship_lo) & (s <= p.ship_hi) & (d >= p.disc_lo) & (d <= p.disc_hi) & (q >= p.qty_lo)
        & (q <= p.qty_hi);
}

// step 1; also clears the output and the meta words for the later steps
__global__ void __launch_bounds__(LK_THREADS) k_li_keys(LiCols c, velo_lineitem_pred p, size_t n, size_t h,
                                                        uint32_t* keys, uint32_t* n_pass, uint32_t* n_ffff, int64_t* out,
                                                        int n_out, LkMeta* meta)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_keys"));
    __shared__ uint32_t tmp[33];
    if (blockIdx.x == 0) {
        if ((int)threadIdx.x < n_out)
            out[threadIdx.x] = 0;
        if (threadIdx.x < SEG_MAX_G)
            meta->slot[threadIdx.x] = 0;
    }
    uint32_t pass = 0, ffff = 0;
    for (size_t i = blockIdx.x * (size_t)LK_THREADS + threadIdx.x; VELO_GRID_COND(i, h);
         i += (size_t)gridDim.x * LK_THREADS) {
        uint32_t w = 0;
#pragma unroll
        for (int lane = 0; lane < 2; lane++) {
            const size_t g = lane ? i + h : i;
            uint32_t k = LK_NONE;
            if (g < n) {
                VELO_TRACE_AT(TS_LI_IN, c.qty + g);
                const bool ok = li_pass(c, p, g);
                const uint32_t key = ((uint32_t)c.f1[g] << 8) | c.f2[g];
                k = ok ? key : LK_NONE;
                pass += ok ? 1u : 0u;
                ffff += (ok & (key == LK_NONE)) ? 1u : 0u;
            }
            w |= k << (16 * lane);
        }
        VELO_TRACE_AT(TS_LI_OUT, keys + i);
        keys[i] = w;
    }
    uint32_t t0, t1;
    block_exclusive_scan(pass, tmp, &t0);
    block_exclusive_scan(ffff, tmp, &t1);
    if (threadIdx.x == 0) {
        n_pass[blockIdx.x] = t0;
        n_ffff[blockIdx.x] = t1;
    }
}

// out word i = (min, max) of the low lane at i and the high lane at N - 1 - i,
// rows from h on being padding
__global__ void __launch_bounds__(LK_THREADS) k_li_fold(const uint32_t* in, size_t h, size_t N, uint32_t* out)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_fold"));
    for (size_t i = blockIdx.x * (size_t)LK_THREADS + threadIdx.x; VELO_GRID_COND(i, N);
         i += (size_t)gridDim.x * LK_THREADS) {
        const size_t r = N - 1 - i;
        const uint32_t a = i < h ? in[i] & 0xFFFFu : LK_NONE;
        const uint32_t b = r < h ? in[r] >> 16 : LK_NONE;
        VELO_TRACE_AT(TS_LI_OUT, out + i);
        out[i] = (a < b ? a : b) | ((a < b ? b : a) << 16);
    }
}

// Is the key of lane `lane` at word i the first of its value?  The high lane
// continues the low one: its first key follows the low lane's last.
struct LkTile {
    uint32_t w[LK_TS / LK_THREADS];
    uint32_t prev; // word before the thread's first one
};

// thread t's words t * 16 .. t * 16 + 15 of tile `blk`, through shared memory
// (padded against bank conflicts: 17 words a thread)
__device__ __forceinline__ void lk_load(const uint32_t* keys, size_t N, size_t blk, uint32_t* sm, LkTile& t)
{
    constexpr int R = LK_TS / LK_THREADS;
    const size_t base = blk * LK_TS;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int i = r * LK_THREADS + (int)threadIdx.x;
        VELO_TRACE_AT(TS_SEG_LOAD, keys + base + i);
        sm[i + i / R] = keys[base + i];
    }
    __syncthreads();
    const int i0 = (int)threadIdx.x * R;
#pragma unroll
    for (int r = 0; r < R; r++)
        t.w[r] = sm[i0 + r + (int)threadIdx.x];
    if (threadIdx.x > 0)
        t.prev = sm[i0 - 1 + (i0 - 1) / R];
    else if (blk > 0)
        t.prev = keys[base - 1];
    else // nothing before the low lane; the low lane's last key before the high lane
        t.prev = keys[N - 1] << 16;
    __syncthreads();
    if (threadIdx.x == 0 && blk == 0)
        t.prev = (t.prev & 0xFFFF0000u) | (~t.w[0] & 0xFFFFu); // differs from the first key
}

// step 3a: first occurrences of each tile, low and high lane
__global__ void __launch_bounds__(LK_THREADS) k_li_distinct(const uint32_t* keys, size_t N, uint32_t* cnt0,
                                                            uint32_t* cnt1)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_distinct"));
    __shared__ uint32_t sm[LK_TS + LK_THREADS];
    __shared__ uint32_t tmp[33];
    LkTile t;
    lk_load(keys, N, blockIdx.x, sm, t);
    uint32_t p = t.prev, c0 = 0, c1 = 0;
#pragma unroll
    for (int r = 0; r < LK_TS / LK_THREADS; r++) {
        const uint32_t x = t.w[r] ^ p;
        c0 += ((x & 0xFFFFu) != 0 && (t.w[r] & 0xFFFFu) != LK_NONE) ? 1u : 0u;
        c1 += ((x >> 16) != 0 && (t.w[r] >> 16) != LK_NONE) ? 1u : 0u;
        p = t.w[r];
    }
    uint32_t t0, t1;
    block_exclusive_scan(c0, tmp, &t0);
    block_exclusive_scan(c1, tmp, &t1);
    if (threadIdx.x == 0) {
        VELO_TRACE_AT(TS_SEG_META, cnt0 + blockIdx.x);
        cnt0[blockIdx.x] = t0;
        cnt1[blockIdx.x] = t1;
    }
}

// sum of x[0 .. n) over the CTA, all threads; tmp: 33 words
__device__ __forceinline__ uint32_t lk_sum(const uint32_t* x, int n, uint32_t* tmp)
{
    uint32_t s = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        VELO_TRACE_AT(TS_SEG_META, x + i);
        s += x[i];
    }
    uint32_t total;
    block_exclusive_scan(s, tmp, &total);
    return total;
}

// step 3b: the first G first occurrences become the slots
__global__ void __launch_bounds__(LK_THREADS) k_li_slots(const uint32_t* keys, size_t N, int ntiles,
                                                         const uint32_t* cnt0, const uint32_t* cnt1,
                                                         const uint32_t* n_pass, const uint32_t* n_ffff, int nblk, int G,
                                                         LkMeta* meta)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_slots"));
    __shared__ uint32_t sm[LK_TS + LK_THREADS];
    __shared__ uint32_t tmp[33];
    __shared__ uint32_t s_slot[SEG_MAX_G];
    constexpr int R = LK_TS / LK_THREADS;
    const int blk = (int)blockIdx.x;
    LkTile t;
    lk_load(keys, N, blk, sm, t);
    if (threadIdx.x < SEG_MAX_G)
        s_slot[threadIdx.x] = 0;
    uint32_t f0 = 0, f1 = 0, p = t.prev; // bit r: the thread's word r holds a first occurrence
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t x = t.w[r] ^ p;
        f0 |= ((x & 0xFFFFu) != 0 && (t.w[r] & 0xFFFFu) != LK_NONE) ? 1u << r : 0u;
        f1 |= ((x >> 16) != 0 && (t.w[r] >> 16) != LK_NONE) ? 1u << r : 0u;
        p = t.w[r];
    }
    uint32_t total;
    const uint32_t ex0 = block_exclusive_scan(__popc(f0), tmp, &total);
    const uint32_t ex1 = block_exclusive_scan(__popc(f1), tmp, &total);
    const uint32_t all0 = lk_sum(cnt0, ntiles, tmp);
    const uint32_t rank0 = lk_sum(cnt0, blk, tmp) + ex0;
    const uint32_t rank1 = all0 + lk_sum(cnt1, blk, tmp) + ex1;
    for (int j = 0; j < G; j++) {
        uint32_t v = 0, r0 = rank0, r1 = rank1;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const bool a = (f0 >> r) & 1u, b = (f1 >> r) & 1u;
            v |= (a & (r0 == (uint32_t)j)) ? (t.w[r] & 0xFFFFu) + 1u : 0u;
            v |= (b & (r1 == (uint32_t)j)) ? (t.w[r] >> 16) + 1u : 0u;
            r0 += a ? 1u : 0u;
            r1 += b ? 1u : 0u;
        }
        v = __reduce_or_sync(0xFFFFFFFFu, v);
        if ((threadIdx.x & 31) == 0)
            atomicOr(&s_slot[j], v);
    }
    if (blk == 0) {
        // the groups and rows in all; 0xFFFF, which the sort took for a row
        // that fails, is the last group if a passing row has it
        const uint32_t distinct = all0 + lk_sum(cnt1, ntiles, tmp);
        const uint32_t ffff = lk_sum(n_ffff, nblk, tmp);
        uint64_t rows = 0;
        for (int i = threadIdx.x; i < nblk; i += LK_THREADS)
            rows += n_pass[i];
        rows = (uint64_t)warp_sum_i64((int64_t)rows);
        __shared__ unsigned long long s_rows;
        if (threadIdx.x == 0)
            s_rows = 0;
        __syncthreads();
        if ((threadIdx.x & 31) == 0)
            atomicAdd(&s_rows, (unsigned long long)rows);
        __syncthreads();
        if (threadIdx.x < SEG_MAX_G && ffff != 0 && distinct == threadIdx.x)
            s_slot[threadIdx.x] = LK_NONE + 1u;
        if (threadIdx.x == 0) {
            meta->rows = s_rows;
            meta->groups = (uint64_t)distinct + (ffff != 0 ? 1u : 0u);
        }
    }
    __syncthreads();
    // one update per CTA and slot at a fixed address
    if ((int)threadIdx.x < G)
        atomicOr(&meta->slot[threadIdx.x], s_slot[threadIdx.x]);
}

// Step 4: rows of this CTA's grid stride into slots 8 * blockIdx.y .. + 7.
// Bound by the integer pipes (about 10 predicated additions a row and slot)
// and HBM (26 bytes a row).
constexpr int LK_SLOTS = 8;
__global__ void __launch_bounds__(LK_THREADS, 2) k_li_sums(LiCols c, velo_lineitem_pred p, size_t n, int G,
                                                          const LkMeta* meta, int64_t* out, uint64_t* d_counts)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_sums"));
    __shared__ int64_t red[LK_THREADS / 32][LK_SLOTS * LI_V];
    const int j0 = (int)blockIdx.y * LK_SLOTS;
    uint32_t slot[LK_SLOTS];
    int64_t acc[LK_SLOTS][LI_V];
#pragma unroll
    for (int j = 0; j < LK_SLOTS; j++) {
        slot[j] = j0 + j < G ? meta->slot[j0 + j] : 0u;
#pragma unroll
        for (int v = 0; v < LI_V; v++)
            acc[j][v] = 0;
    }
    const size_t stride = (size_t)gridDim.x * LK_THREADS;
#pragma unroll 2
    for (size_t g = blockIdx.x * (size_t)LK_THREADS + threadIdx.x; VELO_GRID_COND(g, n); g += stride) {
        VELO_TRACE_AT(TS_LI_IN, c.qty + g);
        const int32_t q = c.qty[g], d = c.disc[g], t = c.tax[g], s = c.ship[g];
        const int64_t price = c.price[g];
        const uint32_t key = ((uint32_t)c.f1[g] << 8) | c.f2[g];
        const bool ok = (s >= p.ship_lo) & (s <= p.ship_hi) & (d >= p.disc_lo) & (d <= p.disc_hi) & (q >= p.qty_lo)
            & (q <= p.qty_hi);
        const uint32_t k1 = ok ? key + 1u : ~0u; // no slot holds ~0
        const int64_t dp = price * (100 - (int64_t)d);
        const int64_t ch = dp * (100 + (int64_t)t);
#pragma unroll
        for (int j = 0; j < LK_SLOTS; j++) {
            const bool hit = slot[j] == k1;
            acc[j][0] += hit ? 1 : 0;
            acc[j][1] += hit ? (int64_t)q : 0;
            acc[j][2] += hit ? price : 0;
            acc[j][3] += hit ? dp : 0;
            acc[j][4] += hit ? ch : 0;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < LK_SLOTS; j++)
#pragma unroll
        for (int v = 0; v < LI_V; v++) {
            const int64_t s = warp_sum_i64(acc[j][v]);
            if (lane == 0)
                red[warp][j * LI_V + v] = s;
        }
    __syncthreads();
    for (int q = threadIdx.x; q < LK_SLOTS * LI_V; q += LK_THREADS) {
        const int j = j0 + q / LI_V, v = q % LI_V;
        if (j < G) {
            int64_t s = 0;
#pragma unroll
            for (int w = 0; w < LK_THREADS / 32; w++)
                s += red[w][q];
            VELO_TRACE_AT(TS_SEG_OUT, out + j * (1 + LI_V) + 1 + v);
            atomicAdd(reinterpret_cast<unsigned long long*>(out + j * (1 + LI_V) + 1 + v), (unsigned long long)s);
        }
    }
    if (blockIdx.x == 0) {
        if ((int)threadIdx.x < LK_SLOTS && j0 + (int)threadIdx.x < G) {
            const uint32_t k = meta->slot[j0 + threadIdx.x];
            out[(j0 + threadIdx.x) * (1 + LI_V)] = k ? (int64_t)(k - 1u) : 0;
        }
        if (blockIdx.y == 0 && threadIdx.x == 0) {
            d_counts[0] = meta->rows;
            d_counts[1] = meta->groups;
        }
    }
}

static velo_status run_groupby(const LiScratch& s, const LiCols& c, size_t n, const velo_lineitem_pred& pred,
                               uint32_t group_bound, int64_t* d_out, uint64_t* d_counts, cudaStream_t st)
{
    const int G = (int)group_bound;
    const size_t h = (n + 1) / 2;
    const int logH = ilog2_floor(next_pow2(h));
    // the merged keys: a power of two of whole tiles
    const int logN = logH < LK_LT ? LK_LT : logH;
    const size_t N = (size_t)1 << logN;
    // scratch: the key words in w[0], the merged ones from w[1] on (w[1] and
    // w[2] are adjacent and hold 16 bytes a row of at least 4096 rows); the
    // count arrays in the tile arrays of the record pipeline
    uint32_t* ka = reinterpret_cast<uint32_t*>(s.w[0]);
    uint32_t* kb = reinterpret_cast<uint32_t*>(s.w[1]);
    const int ntiles = (int)(N / LK_TS);
    uint32_t* cnt0 = s.counts;
    uint32_t* cnt1 = s.counts + ntiles;
    uint32_t* n_pass = s.prefix;
    uint32_t* n_ffff = s.tail_prefix;
    LkMeta* meta = reinterpret_cast<LkMeta*>(s.d_rows);
    StageTimer tm(st);

    // 1. keys
    const size_t want = (h + LK_ROWS - 1) / LK_ROWS;
    const unsigned nblk = want < LK_MAX_BLOCKS ? (unsigned)want : LK_MAX_BLOCKS;
    k_li_keys<<<nblk, LK_THREADS, 0, st>>>(c, pred, n, h, ka, n_pass, n_ffff, d_out, G * (1 + LI_V), meta);
    VELO_CUDA_TRY(cudaGetLastError(), "group-by keys launch");
    tm.mark();
    // 2. sort both lanes, fold, merge
    if (h > 1) {
        std::vector<NetPass> passes;
        plan_sort(logH, LK_LT, LK_LMAX, passes);
        const velo_status rc = launch_net<RowU2, LK_LOG_NT, LK_LOG_E>(
            RowU2::Cols { ka }, NetGeom::trimmed(h, logH, LK_LT, 0), passes, nullptr, st);
        if (rc != VELO_OK)
            return rc;
    }
    k_li_fold<<<(unsigned)(N / LK_ROWS < LK_MAX_BLOCKS ? N / LK_ROWS : LK_MAX_BLOCKS), LK_THREADS, 0, st>>>(ka, h, N,
                                                                                                       kb);
    VELO_CUDA_TRY(cudaGetLastError(), "group-by fold launch");
    {
        std::vector<NetPass> passes;
        plan_merge(logN, LK_LT, LK_LMAX, logN, passes);
        const velo_status rc =
            launch_net<RowU2, LK_LOG_NT, LK_LOG_E>(RowU2::Cols { kb }, NetGeom(N, logN), passes, nullptr, st);
        if (rc != VELO_OK)
            return rc;
    }
    tm.mark();
    // 3. the groups' keys in order
    k_li_distinct<<<ntiles, LK_THREADS, 0, st>>>(kb, N, cnt0, cnt1);
    k_li_slots<<<ntiles, LK_THREADS, 0, st>>>(kb, N, ntiles, cnt0, cnt1, n_pass, n_ffff, (int)nblk, G, meta);
    VELO_CUDA_TRY(cudaGetLastError(), "group-by slots launch");
    tm.mark();
    // 4. masked sums
    const size_t wb = (n + LK_ROWS - 1) / LK_ROWS;
    const dim3 grid((unsigned)(wb < 148 * 2 ? wb : 148 * 2), (unsigned)((G + LK_SLOTS - 1) / LK_SLOTS));
    k_li_sums<<<grid, LK_THREADS, 0, st>>>(c, pred, n, G, meta, d_out, d_counts);
    VELO_CUDA_TRY(cudaGetLastError(), "group-by sums launch");
    tm.mark();
    tm.finish();
    return VELO_OK;
}

} // namespace velo

using namespace velo;

extern "C" size_t velo_filter_groupby_scratch_bytes(size_t n, uint32_t group_bound)
{
    if (group_bound == 0 || group_bound > SEG_MAX_G)
        return 0;
    return li_layout(nullptr, n, group_bound).bytes;
}

extern "C" velo_status velo_filter_groupby(const velo_lineitem* cols, size_t n, const velo_lineitem_pred* pred,
                                           uint32_t group_bound, uint32_t flags, int64_t* d_out, uint64_t* d_counts,
                                           void* d_scratch, size_t scratch_bytes, void* stream)
{
    if (!cols || !pred || !d_out || !d_counts)
        return einval("velo_filter_groupby: null argument");
    if (group_bound == 0 || group_bound > SEG_MAX_G)
        return einval("velo_filter_groupby: group_bound must be 1..16");
    if (n == 0 || next_pow2(n) > ((size_t)1 << MAX_LOGN))
        return einval("velo_filter_groupby: n must be 1..2^31");
    if (!cols->qty || !cols->price || !cols->disc || !cols->tax || !cols->shipdate || !cols->flag1 || !cols->flag2)
        return einval("velo_filter_groupby: null column");
    LiScratch s = li_layout(static_cast<char*>(d_scratch), n, group_bound);
    if (!d_scratch || scratch_bytes < s.bytes) {
        set_error("velo_filter_groupby: scratch must hold velo_filter_groupby_scratch_bytes() bytes");
        return VELO_ENOMEM;
    }
    cudaStream_t st = (cudaStream_t)stream;
    LiCols c { cols->qty, cols->price, cols->disc, cols->tax, cols->shipdate, cols->flag1, cols->flag2 };
    (void)flags; // no step reads the filtered count back, revealed or not
    return run_groupby(s, c, n, *pred, group_bound, d_out, d_counts, st);
}
