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
//               lane (with VELO_REVEAL_COUNT and few rows passing, of the words
//               that hold such a row: reveal_words)
//   3. groups   rows whose key differs from the one before are the groups, in
//               key order; a prefix count ranks them and each of the first
//               group_bound becomes a slot
//   4. sums     every row is added to every slot with a mask (exact int64)
// It replaces FilterCompactionOperator's scatter/gather
// (src/operator/filter_compaction_operator.cpp:65-184) and the sorted
// segmented sums of obliviator/operator_2/enclave/
// scalable_oblivious_join.c:221-262: the same groups, counts and sums.  The
// order of the passes and every address depend on n, group_bound and, only where
// it is revealed, the number of passing rows.
//
// Why: sorting 16-byte records of next_pow2(n) rows took 1.74 ms of a 2.17 ms
// call at 6,001,215 rows (ORCompact 0.31 ms, aggregation 0.29 ms).  The keys
// are an eighth of the bytes, an exchange of two keys is four instructions
// instead of two exchanges of about 19, and the rows' 26 bytes are read once
// here.  6,001,215 rows: 2,166 -> 421 us (its stages one after another: keys 23,
// sort 279, groups 40, sums 92).
#include "net_host.cuh"
#include "groupby.cuh"

namespace velo {

// log2 of the key words a tile holds, 256 threads of 8, 16 or 32 words, for the
// network over 2^log_words of them.  One tile of up to 4096 words is no larger than
// it has to be (a call of 5,000 rows 59 -> 47 us).  Beyond that smaller tiles shorten
// a call, but their passes are more work: with the count revealed, where a call
// waits for its own result, 2048 words up to 2^18 and 4096 up to 2^21 (with 11 / 12 /
// 13, us, 8 groups: 12,000 rows 60 / 67 / 71, 70,001 78 / 86 / 107, 300,000 92 / 100 /
// 129, 1 M 138 / 131 / 146, 3 M 281 / 256 / 261, 6 M 542 / 436 / 421); else 8192, which
// serves more queries a second on several streams (16 streams, 2^14..2^18 rows:
// 12,400 against 11,700).
static int lk_lt(int log_words, bool reveal)
{
    if (log_words <= 12)
        return log_words <= 11 ? 11 : 12;
    return !reveal || log_words > 21 ? 13 : log_words <= 18 ? 11 : 12;
}
constexpr unsigned LK_MAX_BLOCKS = 148 * 8;
// the sums: 8 slots a thread take 72 registers of sums
constexpr int LK_SLOTS = 8, LKS_THREADS = 128, LKS_CTAS = 3;

__global__ void __launch_bounds__(LK_THREADS) k_li_keys(LiCols c, velo_lineitem_pred p, size_t n, LkPlan q, int64_t* out,
                                                        int n_out)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_keys"));
    __shared__ uint32_t tmp[33];
    li_keys_body(c, p, n, q.h, q.ka, q.n_pass, q.n_ffff, out, n_out, q.meta, blockIdx.x, gridDim.x, tmp);
}

__global__ void __launch_bounds__(LK_THREADS) k_li_fold(LkPlan q)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_fold"));
    li_fold_body(q.ka, q.h, q.N, q.kb, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(LK_THREADS) k_li_distinct(LkPlan q)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_distinct"));
    __shared__ uint32_t sm[LK_SM];
    __shared__ uint32_t tmp[33];
    li_distinct_tile(q.kb, q.N, q.cnt0, q.cnt1, blockIdx.x, sm, tmp);
}

__global__ void __launch_bounds__(LK_THREADS) k_li_slots(LkPlan q, int G)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_slots"));
    __shared__ uint32_t sm[LK_SM];
    __shared__ LkSlotShared x;
    li_slots_tile(q.kb, q.N, q.ntiles, q.cnt0, q.cnt1, q.n_pass, q.n_ffff, (int)q.nblk, G, q.meta, (int)blockIdx.x, sm, x);
}

// Bound by the integer pipes (9 predicated additions a row and slot) and HBM
// (26 bytes a row).
__global__ void __launch_bounds__(LKS_THREADS, LKS_CTAS) k_li_sums(LiCols c, velo_lineitem_pred p, size_t n, int G,
                                                                  const LkMeta* meta, int64_t* out, uint64_t* d_counts)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_sums"));
    __shared__ int64_t red[LKS_THREADS / 32 * LK_SLOTS * LI_V];
    li_sums_body<LK_SLOTS, LKS_THREADS>(c, p, n, G, meta, out, d_counts, (int)blockIdx.y, blockIdx.x, gridDim.x, red);
}

// the sort of h key words, or the last merge of 2^logN words
static velo_status lk_net(uint32_t* keys, size_t h, int logN, bool merge, bool reveal, cudaStream_t st)
{
    const int lt = lk_lt(logN, reveal);
    std::vector<NetPass> passes;
    if (merge)
        plan_merge(logN, lt, lt - 4, logN, passes);
    else
        plan_sort(logN, lt, lt - 4, passes);
    const RowU2::Cols c { keys };
    const NetGeom g = merge ? NetGeom(h, logN) : NetGeom::trimmed(h, logN, lt, 0);
    return lt == 11 ? launch_net<RowU2, 8, 3>(c, g, passes, nullptr, st)
        : lt == 12  ? launch_net<RowU2, 8, 4>(c, g, passes, nullptr, st)
                    : launch_net<RowU2, 8, 5>(c, g, passes, nullptr, st);
}

// the number of passing rows, by one CTA
__global__ void __launch_bounds__(1024) k_li_rows(LkPlan q)
{
    VELO_TRACE_KERNEL(velo_site_hash("k_li_rows"));
    __shared__ uint32_t tmp[33];
    const uint32_t rows = lk_sum(q.n_pass, (int)q.nblk, tmp);
    if (threadIdx.x == 0)
        q.meta->rows = rows;
}

// With the count revealed (VELO_REVEAL_COUNT): when next_pow2(rows passing) is at
// most half of the 2^logH key words, the words that hold such a row are compacted
// to the front and `rows` words are sorted in the place of all h.  The count
// costs a copy to the host (about 17 us), so calls of at most 2^18 words, whose
// whole sort takes 45 us and less in small tiles, do without it.
// Revealed / not / 16-byte records compacted and sorted (us, 8 groups), 2 % of the
// rows passing: 600,000 rows 113 / 142 / 133, 1 M 119 / 146 / 145, 3 M 172 / 258 /
// 250, 6,001,215 262 / 420 / 405; 0.2 %: 94 / 146 / 109 at 1 M; 50 %: 435 / 420 /
// 1,087 at 6,001,215.
constexpr int LK_REVEAL_LOGH = 19;

static velo_status reveal_words(const LiScratch& s, LkPlan& q, cudaStream_t st)
{
    // a stream that is being captured cannot be waited for
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    VELO_CUDA_TRY(cudaStreamIsCapturing(st, &cap), "cudaStreamIsCapturing");
    if (cap != cudaStreamCaptureStatusNone)
        return VELO_OK;
    k_li_rows<<<1, 1024, 0, st>>>(q);
    VELO_CUDA_TRY(cudaGetLastError(), "group-by count launch");
    uint64_t rows = 0;
    VELO_CUDA_TRY(cudaMemcpyAsync(&rows, &q.meta->rows, 8, cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync");
    VELO_CUDA_TRY(cudaStreamSynchronize(st), "cudaStreamSynchronize");
    if (next_pow2(rows ? rows : 1) > (size_t)1 << (q.logH - 1))
        return VELO_OK;
    const RowW::Cols c { q.ka };
    const int lt = q.logH <= 20 ? LK_COMPACT_LT : 13;
    velo_status rc = launch_count_scan<RowW>(c, q.h, q.logH, lt, s.tile_counts, s.tile_prefix, nullptr, st);
    if (rc != VELO_OK)
        return rc;
    std::vector<NetPass> passes;
    plan_compact(q.logH, lt, 9, passes); // (8 or 16 words a segment)
    const NetGeom g(q.h, q.logH);
    rc = lt == LK_COMPACT_LT ? launch_net<RowW, 8, 4>(c, g, passes, s.tile_prefix, st)
                             : launch_net<RowW, 8, 5>(c, g, passes, s.tile_prefix, st);
    if (rc == VELO_OK)
        lk_words(q, s, rows ? rows : 1, 12);
    return rc;
}

static velo_status run_groupby(const LiScratch& s, const LiCols& c, size_t n, const velo_lineitem_pred& pred,
                               uint32_t group_bound, bool reveal, int64_t* d_out, uint64_t* d_counts, cudaStream_t st)
{
    const int G = (int)group_bound;
    LkPlan q = lk_plan(s, n, 12, LK_MAX_BLOCKS);
    StageTimer tm(st);

    // 1. keys
    k_li_keys<<<q.nblk, LK_THREADS, 0, st>>>(c, pred, n, q, d_out, G * (1 + LI_V));
    VELO_CUDA_TRY(cudaGetLastError(), "group-by keys launch");
    tm.mark();
    // 2. sort both lanes, fold, merge
    if (reveal && q.logH >= LK_REVEAL_LOGH) {
        const velo_status rc = reveal_words(s, q, st);
        if (rc != VELO_OK)
            return rc;
    }
    if (q.h > 1) {
        const velo_status rc = lk_net(q.ka, q.h, q.logH, false, reveal, st);
        if (rc != VELO_OK)
            return rc;
    }
    k_li_fold<<<(unsigned)(q.N / LK_ROWS < LK_MAX_BLOCKS ? q.N / LK_ROWS : LK_MAX_BLOCKS), LK_THREADS, 0, st>>>(q);
    VELO_CUDA_TRY(cudaGetLastError(), "group-by fold launch");
    {
        const velo_status rc = lk_net(q.kb, q.N, q.logN, true, reveal, st);
        if (rc != VELO_OK)
            return rc;
    }
    tm.mark();
    // 3. the groups' keys in order
    if (q.ntiles > 1)
        k_li_distinct<<<q.ntiles, LK_THREADS, 0, st>>>(q);
    k_li_slots<<<q.ntiles, LK_THREADS, 0, st>>>(q, G);
    VELO_CUDA_TRY(cudaGetLastError(), "group-by slots launch");
    tm.mark();
    // 4. masked sums
    const size_t wb = (n + LK_ROWS - 1) / LK_ROWS;
    const dim3 grid((unsigned)(wb < 148 * LKS_CTAS ? wb : 148 * LKS_CTAS), (unsigned)((G + LK_SLOTS - 1) / LK_SLOTS));
    k_li_sums<<<grid, LKS_THREADS, 0, st>>>(c, pred, n, G, q.meta, d_out, d_counts);
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
    return run_groupby(s, c, n, *pred, group_bound, (flags & VELO_REVEAL_COUNT) != 0, d_out, d_counts, st);
}
