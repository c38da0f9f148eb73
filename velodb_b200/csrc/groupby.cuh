// Filter + group-by over a lineitem-shaped fact table: the steps of the query
// as device bodies, its scratch layout and its geometry, shared by the plain
// pipeline (groupby.cu, where the query is described) and the persistent
// command queue (dq_kernel.cu).  Every body runs on CTAs of LK_THREADS threads
// except the sums, and handles block `blk` of `nblk`.
#pragma once

#include "common.hpp"
#include "network.cuh"
#include "segagg.cuh"

namespace velo {

// output values of a group: count, sum qty, sum price, sum price*(100-disc),
// sum price*(100-disc)*(100+tax)
constexpr int LI_V = 5;

struct LiCols {
    const int32_t* qty;
    const int64_t* price;
    const int32_t* disc;
    const int32_t* tax;
    const int32_t* ship;
    const uint8_t* f1;
    const uint8_t* f2;
};

constexpr int LK_THREADS = 256;
constexpr int LK_ROWS = 1024; // key words of a block's first grid-stride step
constexpr int LK_TS = 4096;   // key words of a tile of the group search
constexpr int LK_LMAX = 9;
constexpr uint32_t LK_NONE = 0xFFFFu;

// the words the later steps share
struct LkMeta {
    uint64_t rows;            // rows passing the filter
    uint64_t groups;          // distinct keys among them
    uint32_t slot[SEG_MAX_G]; // key + 1 of group j, 0 past the last group
};

__device__ __forceinline__ bool li_pass(const velo_lineitem_pred& p, int32_t q, int32_t d, int32_t s)
{
    return (s >= p.ship_lo) & (s <= p.ship_hi) & (d >= p.disc_lo) & (d <= p.disc_hi) & (q >= p.qty_lo)
        & (q <= p.qty_hi);
}

// step 1: key words, rows passing and rows passing with the key 0xFFFF; also
// clears the output and the slots for the later steps.  tmp: 33 words
__device__ __forceinline__ void li_keys_body(const LiCols& c, const velo_lineitem_pred& p, size_t n, size_t h,
                                             uint32_t* keys, uint32_t* n_pass, uint32_t* n_ffff, int64_t* out,
                                             int n_out, LkMeta* meta, size_t blk, size_t nblk, uint32_t* tmp)
{
    if (blk == 0) {
        if ((int)threadIdx.x < n_out)
            out[threadIdx.x] = 0;
        if (threadIdx.x < SEG_MAX_G)
            meta->slot[threadIdx.x] = 0;
    }
    uint32_t pass = 0, ffff = 0;
    for (size_t i = blk * (size_t)LK_THREADS + threadIdx.x; VELO_GRID_COND(i, h);
         i += nblk * (size_t)LK_THREADS) {
        uint32_t w = 0;
#pragma unroll
        for (int lane = 0; lane < 2; lane++) {
            const size_t g = lane ? i + h : i;
            uint32_t k = LK_NONE;
            if (g < n) {
                VELO_TRACE_AT(TS_LI_IN, c.qty + g);
                const bool ok = li_pass(p, c.qty[g], c.disc[g], c.ship[g]);
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
        n_pass[blk] = t0;
        n_ffff[blk] = t1;
    }
}

// out word i = (min, max) of the low lane at i and the high lane at N - 1 - i,
// rows from h on being padding
__device__ __forceinline__ void li_fold_body(const uint32_t* in, size_t h, size_t N, uint32_t* out, size_t blk,
                                             size_t nblk)
{
    for (size_t i = blk * (size_t)LK_THREADS + threadIdx.x; VELO_GRID_COND(i, N);
         i += nblk * (size_t)LK_THREADS) {
        const size_t r = N - 1 - i;
        if (i < h)
            VELO_TRACE_AT(TS_LI_IN, in + i);
        if (r < h)
            VELO_TRACE_AT(TS_LI_IN, in + r);
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

// step 3a: first occurrences of each tile, low and high lane.  sm: LK_SM words,
// tmp: 33 words
constexpr int LK_SM = LK_TS + LK_THREADS;
__device__ __forceinline__ void li_distinct_tile(const uint32_t* keys, size_t N, uint32_t* cnt0, uint32_t* cnt1,
                                                 size_t blk, uint32_t* sm, uint32_t* tmp)
{
    LkTile t;
    lk_load(keys, N, blk, sm, t);
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
        VELO_TRACE_AT(TS_SEG_META, cnt0 + blk);
        cnt0[blk] = t0;
        cnt1[blk] = t1;
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

// step 3b: the first G first occurrences become the slots (one tile counts its
// own, without step 3a).  sm: LK_SM words
struct LkSlotShared {
    unsigned long long rows;
    uint32_t slot[SEG_MAX_G];
    uint32_t tmp[33];
};
__device__ __forceinline__ void li_slots_tile(const uint32_t* keys, size_t N, int ntiles, const uint32_t* cnt0,
                                              const uint32_t* cnt1, const uint32_t* n_pass, const uint32_t* n_ffff,
                                              int nblk, int G, LkMeta* meta, int blk, uint32_t* sm, LkSlotShared& x)
{
    constexpr int R = LK_TS / LK_THREADS;
    LkTile t;
    lk_load(keys, N, blk, sm, t);
    if (threadIdx.x < SEG_MAX_G)
        x.slot[threadIdx.x] = 0;
    uint32_t f0 = 0, f1 = 0, p = t.prev; // bit r: the thread's word r holds a first occurrence
#pragma unroll
    for (int r = 0; r < R; r++) {
        const uint32_t d = t.w[r] ^ p;
        f0 |= ((d & 0xFFFFu) != 0 && (t.w[r] & 0xFFFFu) != LK_NONE) ? 1u << r : 0u;
        f1 |= ((d >> 16) != 0 && (t.w[r] >> 16) != LK_NONE) ? 1u << r : 0u;
        p = t.w[r];
    }
    uint32_t all0, all1;
    const uint32_t ex0 = block_exclusive_scan(__popc(f0), x.tmp, &all0);
    const uint32_t ex1 = block_exclusive_scan(__popc(f1), x.tmp, &all1);
    uint32_t rank0 = ex0;
    uint32_t rank1 = ex1;
    if (ntiles > 1) {
        all0 = lk_sum(cnt0, ntiles, x.tmp);
        rank0 += lk_sum(cnt0, blk, x.tmp);
        rank1 += lk_sum(cnt1, blk, x.tmp);
    }
    rank1 += all0;
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
            atomicOr(&x.slot[j], v);
    }
    if (blk == 0) {
        // the groups and rows in all; 0xFFFF, which the sort took for a row
        // that fails, is the last group if a passing row has it
        const uint32_t distinct = all0 + (ntiles > 1 ? lk_sum(cnt1, ntiles, x.tmp) : all1);
        const uint32_t ffff = lk_sum(n_ffff, nblk, x.tmp);
        uint64_t rows = 0;
        for (int i = threadIdx.x; i < nblk; i += LK_THREADS)
            rows += n_pass[i];
        rows = (uint64_t)warp_sum_i64((int64_t)rows);
        if (threadIdx.x == 0)
            x.rows = 0;
        __syncthreads();
        if ((threadIdx.x & 31) == 0)
            atomicAdd(&x.rows, (unsigned long long)rows);
        __syncthreads();
        if (threadIdx.x < SEG_MAX_G && ffff != 0 && distinct == threadIdx.x)
            x.slot[threadIdx.x] = LK_NONE + 1u;
        if (threadIdx.x == 0) {
            meta->rows = x.rows;
            meta->groups = (uint64_t)distinct + (ffff != 0 ? 1u : 0u);
        }
    }
    __syncthreads();
    // one update per CTA and slot at a fixed address
    if ((int)threadIdx.x < G)
        atomicOr(&meta->slot[threadIdx.x], x.slot[threadIdx.x]);
}

// one row's columns
struct LkRow {
    int32_t q, d, t, s;
    int64_t price;
    uint32_t key;
};
__device__ __forceinline__ LkRow lk_row(const LiCols& c, size_t g)
{
    VELO_TRACE_AT(TS_LI_IN, c.qty + g);
    return LkRow { c.qty[g], c.disc[g], c.tax[g], c.ship[g], c.price[g], ((uint32_t)c.f1[g] << 8) | c.f2[g] };
}

// one slot's sums; a row is added by predicated additions, carries included
// (a select and an addition per half otherwise)
struct LkAcc {
    uint32_t n = 0;
    uint32_t lo[LI_V - 1] = {}, hi[LI_V - 1] = {};
    __device__ __forceinline__ void add(uint32_t slot, uint32_t k, int32_t q, int64_t price, int64_t dp,
                                        int64_t ch)
    {
        asm("{\n\t.reg .pred p;\n\t"
            "setp.eq.u32 p, %9, %18;\n\t"
            "@p add.u32 %0, %0, 1;\n\t"
            "@p add.cc.u32 %1, %1, %10;\n\t"
            "@p addc.u32 %2, %2, %11;\n\t"
            "@p add.cc.u32 %3, %3, %12;\n\t"
            "@p addc.u32 %4, %4, %13;\n\t"
            "@p add.cc.u32 %5, %5, %14;\n\t"
            "@p addc.u32 %6, %6, %15;\n\t"
            "@p add.cc.u32 %7, %7, %16;\n\t"
            "@p addc.u32 %8, %8, %17;\n\t}"
            : "+r"(n), "+r"(lo[0]), "+r"(hi[0]), "+r"(lo[1]), "+r"(hi[1]), "+r"(lo[2]), "+r"(hi[2]), "+r"(lo[3]),
              "+r"(hi[3])
            : "r"(slot), "r"((uint32_t)q), "r"((uint32_t)(q >> 31)), "r"((uint32_t)price),
              "r"((uint32_t)((uint64_t)price >> 32)), "r"((uint32_t)dp), "r"((uint32_t)((uint64_t)dp >> 32)),
              "r"((uint32_t)ch), "r"((uint32_t)((uint64_t)ch >> 32)), "r"(k));
    }
    __device__ __forceinline__ int64_t value(int v) const
    {
        return v == 0 ? (int64_t)n : (int64_t)(((uint64_t)hi[v - 1] << 32) | lo[v - 1]);
    }
};

// Step 4: rows of this block's grid stride into slots SLOTS * chunk .. of NT
// threads; red: (NT / 32) * SLOTS * LI_V words of shared memory
template <int SLOTS, int NT>
__device__ __forceinline__ void li_sums_body(const LiCols& c, const velo_lineitem_pred& p, size_t n, int G,
                                             const LkMeta* meta, int64_t* out, uint64_t* d_counts, int chunk,
                                             size_t blk, size_t nblk, int64_t* red)
{
    const int j0 = chunk * SLOTS;
    uint32_t slot[SLOTS];
    LkAcc acc[SLOTS];
#pragma unroll
    for (int j = 0; j < SLOTS; j++)
        slot[j] = j0 + j < G ? meta->slot[j0 + j] : 0u;
    // the next row's columns are loaded while this one is added
    const size_t stride = nblk * (size_t)NT;
    size_t g = blk * (size_t)NT + threadIdx.x;
    LkRow next = {};
    if (g < n)
        next = lk_row(c, g);
    while (g < n) {
        const LkRow r = next;
        g += stride;
        if (g < n)
            next = lk_row(c, g);
        const bool ok = li_pass(p, r.q, r.d, r.s);
        const uint32_t k1 = ok ? r.key + 1u : ~0u; // no slot holds ~0
        const int64_t dp = r.price * (100 - (int64_t)r.d);
        const int64_t ch = dp * (100 + (int64_t)r.t);
#pragma unroll
        for (int j = 0; j < SLOTS; j++)
            acc[j].add(slot[j], k1, r.q, r.price, dp, ch);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < SLOTS; j++)
#pragma unroll
        for (int v = 0; v < LI_V; v++) {
            const int64_t s = warp_sum_i64(acc[j].value(v));
            if (lane == 0)
                red[warp * SLOTS * LI_V + j * LI_V + v] = s;
        }
    __syncthreads();
    for (int q = threadIdx.x; q < SLOTS * LI_V; q += NT) {
        const int j = j0 + q / LI_V, v = q % LI_V;
        if (j < G) {
            int64_t s = 0;
#pragma unroll
            for (int w = 0; w < NT / 32; w++)
                s += red[w * SLOTS * LI_V + q];
            VELO_TRACE_AT(TS_SEG_OUT, out + j * (1 + LI_V) + 1 + v);
            atomicAdd(reinterpret_cast<unsigned long long*>(out + j * (1 + LI_V) + 1 + v), (unsigned long long)s);
        }
    }
    if (blk == 0) {
        if ((int)threadIdx.x < SLOTS && j0 + (int)threadIdx.x < G) {
            const uint32_t k = meta->slot[j0 + threadIdx.x];
            out[(j0 + threadIdx.x) * (1 + LI_V)] = k ? (int64_t)(k - 1u) : 0;
        }
        if (chunk == 0 && threadIdx.x == 0) {
            d_counts[0] = meta->rows;
            d_counts[1] = meta->groups;
        }
    }
}

struct LiScratch {
    uint32_t* ka;          // key words of step 1, 2^logH words
    uint32_t* kb;          // merged key words, N words
    uint32_t* cnt;         // first occurrences: low lanes, then high lanes of N / LK_TS tiles
    uint32_t *n_pass, *n_ffff; // counts of the blocks of step 1
    uint32_t *tile_counts, *tile_prefix; // marked words of a compaction's tiles and their scan
    LkMeta* meta;
    size_t bytes;
};

constexpr int LK_MIN_LOGN = 13; // merged key words: at least the queue's tile
constexpr int LK_COMPACT_LT = 12; // the smallest tile of a compaction

// What a caller has to bring: the size for the 24-byte records and slot vectors
// that the query used to move.  The steps need a sixth of it; budgets and
// admission by this size stay what they are.
inline size_t li_bytes(size_t n, uint32_t G)
{
    size_t rows = next_pow2(n);
    rows = rows < 4096 ? 4096 : rows;
    const size_t tiles = rows / SEG_TS;
    auto area = [](size_t b) { return align_up(b, 256); };
    return 3 * area(rows * 8) + area(rows / 2048 * 4) + area((rows / 2048 + 1) * 4) + 2 * area(8)
        + area(tiles * sizeof(SegTileAgg)) + 2 * area(tiles * LI_V * 8) + area(tiles * 4)
        + area(tiles * G * (1 + LI_V) * 8);
}

// Partition of the scratch buffer (offsets 256-byte aligned); every area sized
// for the largest geometry that lk_words makes of n rows
inline LiScratch li_layout(char* base, size_t n, uint32_t G)
{
    LiScratch s {};
    const size_t h = (n + 1) / 2;
    const size_t ph = next_pow2(h);
    const size_t N = ph < ((size_t)1 << LK_MIN_LOGN) ? (size_t)1 << LK_MIN_LOGN : ph;
    const size_t nblk = (h + LK_ROWS - 1) / LK_ROWS;
    const size_t ctiles = (ph >> LK_COMPACT_LT) + 1;
    size_t off = 0;
    auto take = [&](size_t words) {
        char* p = base ? base + off : nullptr;
        off += align_up(words * 4, 256);
        return reinterpret_cast<uint32_t*>(p);
    };
    s.ka = take(ph);
    s.kb = take(N);
    s.cnt = take(2 * (N / LK_TS));
    s.n_pass = take(nblk);
    s.n_ffff = take(nblk);
    s.tile_counts = take(ctiles);
    s.tile_prefix = take(ctiles + 1);
    s.meta = reinterpret_cast<LkMeta*>(take((sizeof(LkMeta) + 3) / 4));
    const size_t size = li_bytes(n, G);
    s.bytes = off > size ? off : size;
    return s;
}

// Geometry and scratch of one query with key tiles of 2^lt words
struct LkPlan {
    size_t h; // key words
    int logH;
    size_t N; // merged key words: a power of two of whole tiles
    int logN;
    int ntiles; // tiles of the group search
    unsigned nblk; // blocks of step 1
    uint32_t *ka, *kb, *cnt0, *cnt1, *n_pass, *n_ffff;
    LkMeta* meta;
};

// the key words that are sorted: h of them, merged in tiles of 2^lt words
// (lt <= LK_MIN_LOGN)
inline void lk_words(LkPlan& q, const LiScratch& s, size_t h, int lt)
{
    q.h = h;
    q.logH = ilog2_floor(next_pow2(q.h));
    q.logN = q.logH < lt ? lt : q.logH;
    q.N = (size_t)1 << q.logN;
    q.ntiles = (int)(q.N / LK_TS);
    q.cnt0 = s.cnt;
    q.cnt1 = s.cnt + q.ntiles;
}

inline LkPlan lk_plan(const LiScratch& s, size_t n, int lt, unsigned max_blocks)
{
    LkPlan q {};
    lk_words(q, s, (n + 1) / 2, lt);
    const size_t want = (q.h + LK_ROWS - 1) / LK_ROWS;
    q.nblk = want < max_blocks ? (unsigned)want : max_blocks;
    q.ka = s.ka;
    q.kb = s.kb;
    q.n_pass = s.n_pass;
    q.n_ffff = s.n_ffff;
    q.meta = s.meta;
    return q;
}

} // namespace velo
