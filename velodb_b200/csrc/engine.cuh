// Tile engine for the oblivious networks (bitonic sort, ORCompact) on sm_100a.
//
// A CTA of NT = 2^LOG_NT threads owns a tile of T = 2^t rows (t = LOG_NT +
// LOG_E); every thread keeps E = 2^LOG_E rows in registers.  Which local row
// index a register holds is given by a *layout* s: register e of thread tid
// holds local row
//
//     l = (tid & (2^s - 1)) | (e << s) | ((tid >> s) << (s + LOG_E)),
//
// i.e. the E registers cover local bits [s, s + LOG_E).  A network level whose
// partner bit lies in that window is a register-local compare-exchange; other
// levels first re-layout the tile through shared memory ("transpose", one smem
// write + read of the tile).  Global loads/stores use a layout with s >= 5 so
// the 32 lanes of a warp touch 32 consecutive rows (fully coalesced).
//
// Global loads use ld.global.cg (cached in L2 only): within one persistent
// launch a pass reads rows that other SMs wrote in the previous pass, so the
// non-coherent L1 must not serve them.
//
// Every network step is data-independent: the same loads, stores and smem
// accesses happen for any data of the same public size, and exchanges are
// selects, never branches on data.
#pragma once

#include <cstddef>
#include <cstdint>

#include "trace.cuh"
#include "velo_obl.h"

namespace velo {

// ---------------------------------------------------------------------------
// multi-limb unsigned comparison: 0xFFFFFFFF if x > y else 0, from the borrow
// of y - x (limb 0 least significant); one carry chain, no branches
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t gt_mask3(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t y0, uint32_t y1,
                                             uint32_t y2)
{
    uint32_t r;
    asm("{\n\t.reg .u32 t;\n\t"
        "sub.cc.u32 t, %1, %4;\n\t"
        "subc.cc.u32 t, %2, %5;\n\t"
        "subc.cc.u32 t, %3, %6;\n\t"
        "subc.u32 %0, 0, 0;\n\t}"
        : "=r"(r)
        : "r"(y0), "r"(y1), "r"(y2), "r"(x0), "r"(x1), "r"(x2));
    return r;
}

__device__ __forceinline__ uint32_t gt_mask4(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t y0,
                                             uint32_t y1, uint32_t y2, uint32_t y3)
{
    uint32_t r;
    asm("{\n\t.reg .u32 t;\n\t"
        "sub.cc.u32 t, %1, %5;\n\t"
        "subc.cc.u32 t, %2, %6;\n\t"
        "subc.cc.u32 t, %3, %7;\n\t"
        "subc.cc.u32 t, %4, %8;\n\t"
        "subc.u32 %0, 0, 0;\n\t}"
        : "=r"(r)
        : "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(x0), "r"(x1), "r"(x2), "r"(x3));
    return r;
}

__device__ __forceinline__ uint32_t lo32(uint64_t x) { return (uint32_t)x; }
__device__ __forceinline__ uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }

// 0xFFFFFFFF if the KW-word key x (word 0 most significant) exceeds y
template <int KW>
__device__ __forceinline__ uint32_t key_gt_mask(const uint64_t* x, const uint64_t* y)
{
    if constexpr (KW == 2) {
        return gt_mask4(lo32(x[1]), hi32(x[1]), lo32(x[0]), hi32(x[0]), lo32(y[1]), hi32(y[1]), lo32(y[0]), hi32(y[0]));
    } else {
        // lexicographic from the most significant word
        bool res = false, eq = true;
#pragma unroll
        for (int i = 0; i < KW; i++) {
            res = res | (eq & (x[i] > y[i]));
            eq = eq & (x[i] == y[i]);
        }
        return res ? 0xFFFFFFFFu : 0u;
    }
}

// ---------------------------------------------------------------------------
// row types: SoA columns in global memory, SoA arrays in shared memory.
//
// swap_pred(a, b, desc) is the compare-exchange decision for the pair
// (a at the lower index, b): ascending swaps iff a > b, descending iff a < b.
// STRICT types follow the reference exactly on ties (include/cuda/sort.cuh:
// 31-40: no swap when equal).  Non-strict types are used where the
// arrangement of equal keys is invisible to the consumer (every field is
// compared, or the consumer aggregates over ties); they decide both
// directions with one comparison, swapping equal keys when descending,
// which still sorts.
// ---------------------------------------------------------------------------

template <class T>
__device__ __forceinline__ T sel(bool c, T a, T b)
{
    return c ? a : b;
}

// exchange a and b when x (selects, no branch)
__device__ __forceinline__ void xsel(bool x, uint32_t& a, uint32_t& b)
{
    const uint32_t na = x ? b : a, nb = x ? a : b;
    a = na;
    b = nb;
}

__device__ __forceinline__ void xsel(bool x, uint64_t& a, uint64_t& b)
{
    const uint64_t na = x ? b : a, nb = x ? a : b;
    a = na;
    b = nb;
}

// The same exchange on the integer multiply-add (FMA) pipe: with s = 1 to
// swap (mm = -s), d = b - a, a' = a + d*s, b' = b + d*mm, all mod 2^32.  The
// in-tile levels are bound by the integer ALU pipe (two selects a register);
// doing part of each row's registers here lets both pipes work.  `neg` is -1
// known only at run time, so the subtraction stays a multiply-add too.
struct MadSwap {
    uint32_t s, mm, neg;
    __device__ __forceinline__ explicit MadSwap(bool x)
    {
        neg = (uint32_t)(-(int)(blockDim.x != 0u));
        // an opaque copy: knowing mm is 0 or -1, the compiler would turn the
        // multiply-adds back into selects on the ALU pipe
        const uint32_t m0 = x ? 0xFFFFFFFFu : 0u;
        asm("mov.b32 %0, %1;" : "=r"(mm) : "r"(m0));
        s = mm * neg;
    }
    __device__ __forceinline__ void operator()(uint32_t& a, uint32_t& b) const
    {
        const uint32_t d = a * neg + b;
        a = d * s + a;
        b = d * mm + b;
    }
    __device__ __forceinline__ void operator()(uint64_t& a, uint64_t& b) const
    {
        uint32_t al = lo32(a), ah = hi32(a), bl = lo32(b), bh = hi32(b);
        (*this)(al, bl);
        (*this)(ah, bh);
        a = ((uint64_t)ah << 32) | al;
        b = ((uint64_t)bh << 32) | bl;
    }
};

// The exchange with one select and two multiply-adds a register: with
// t = a + b, a' = x ? b : a (ALU pipe), b' = t - a' (FMA pipe, mod 2^32).
// One instruction fewer than MadSwap and the pipes' shares nearly even; `one`
// is 1 known only at run time (CTAs are one-dimensional), so that the sums
// stay multiply-adds.
struct AddSwap {
    uint32_t one, neg;
    bool x;
    __device__ __forceinline__ explicit AddSwap(bool x_) : one(blockDim.y), neg(0u - blockDim.y), x(x_) { }
    __device__ __forceinline__ void operator()(uint32_t& a, uint32_t& b) const
    {
        const uint32_t t = a * one + b;
        const uint32_t na = x ? b : a;
        b = na * neg + t;
        a = na;
    }
    __device__ __forceinline__ void operator()(uint64_t& a, uint64_t& b) const
    {
        uint32_t al = lo32(a), ah = hi32(a), bl = lo32(b), bh = hi32(b);
        (*this)(al, bl);
        (*this)(ah, bh);
        a = ((uint64_t)ah << 32) | al;
        b = ((uint64_t)bh << 32) | bl;
    }
};

// how a RowRec compares its key
enum KeyMode : int {
    KEY_MASKED = 0, // words 0..KW-1, each AND-ed with Cols::mask (runtime)
    KEY_FULL = 1,   // words 0..KW-1 as they are
    KEY_HI32 = 2,   // the high 32 bits of word 0 only (KW == 1)
    KEY_HI96 = 3,   // word 0 and the high 32 bits of word 1 (KW == 2, strict)
};

// 12-byte rows: u64 key, u32 payload.  Registers hold the key as two 32-bit
// halves so exchanges never repack 64-bit values.  Ordered as CM says:
//   K12_ALL      key, then payload (plain sort rows): every field is compared,
//                so the sorted output is unique
//   K12_KEY_TAG  key, then the top bit of the payload, not strict
//   K12_KEY      the key alone, strict; the rows of descending blocks are
//                complemented (Flip), so one compare serves both directions
// As compaction rows they are marked by a clear top bit of the key.
enum K12Order : int { K12_ALL = 0, K12_KEY_TAG = 1, K12_KEY = 2 };

template <int CM>
struct RowK12 {
    uint32_t kl, kh, p;
    struct Cols {
        uint64_t* k;
        uint32_t* p;
    };
    static constexpr int SMEM_BYTES = 16; // one 16-byte slot per row (kl, kh, p, unused)
    static constexpr int SWZ_BITS = 3;
    __device__ __forceinline__ static RowK12 load(const Cols& c, size_t g)
    {
        VELO_TRACE_AT(TS_ROW_LOAD, c.k + g);
        const uint64_t k = __ldcg(c.k + g);
        return RowK12 { lo32(k), hi32(k), __ldcg(c.p + g) };
    }
    __device__ __forceinline__ static void store(const Cols& c, size_t g, const RowK12& r)
    {
        VELO_TRACE_AT(TS_ROW_STORE, c.k + g);
        c.k[g] = ((uint64_t)r.kh << 32) | r.kl;
        c.p[g] = r.p;
    }
    __device__ __forceinline__ static RowK12 pad(const Cols&) { return RowK12 { ~0u, ~0u, ~0u }; }
    __device__ __forceinline__ static void sstore(char* sm, int, int i, const RowK12& r)
    {
        reinterpret_cast<uint4*>(sm)[i] = make_uint4(r.kl, r.kh, r.p, 0u);
    }
    // the same at byte offset `b` = slot * SLOT_BYTES
    static constexpr int SLOT_BYTES = 16;
    __device__ __forceinline__ static void sstore_b(char* sm, int, uint32_t b, const RowK12& r)
    {
        *reinterpret_cast<uint4*>(sm + b) = make_uint4(r.kl, r.kh, r.p, 0u);
    }
    __device__ __forceinline__ static RowK12 sload_b(const char* sm, int, uint32_t b)
    {
        const uint4 x = *reinterpret_cast<const uint4*>(sm + b);
        return RowK12 { x.x, x.y, x.z };
    }
    __device__ __forceinline__ static RowK12 sload(const char* sm, int, int i)
    {
        const uint4 x = reinterpret_cast<const uint4*>(sm)[i];
        return RowK12 { x.x, x.y, x.z };
    }
    __device__ __forceinline__ static bool swap_pred(const RowK12& a, const RowK12& b, bool desc, const Cols&)
    {
        if constexpr (CM == K12_KEY) {
            return (((uint64_t)a.kh << 32) | a.kl) > (((uint64_t)b.kh << 32) | b.kl);
        } else if constexpr (CM == K12_KEY_TAG) {
            // the lowest limb borrows iff a has the tag and b has not
            return (gt_mask3(a.p & 0x80000000u, a.kl, a.kh, b.p | 0x7FFFFFFFu, b.kl, b.kh) != 0u) != desc;
        } else {
            return (gt_mask3(a.p, a.kl, a.kh, b.p, b.kl, b.kh) != 0u) != desc;
        }
    }
    // exchange a and b when x, in place (2^24-row tile sort 538 -> 507 us,
    // merge 104.9 -> 104.3 us against two halves as MadSwap and one by selects)
    __device__ __forceinline__ static void cswap(RowK12& a, RowK12& b, bool x)
    {
        const AddSwap m(x);
        m(a.kl, b.kl);
        m(a.kh, b.kh);
        m(a.p, b.p);
    }
    __device__ __forceinline__ static RowK12 shfl_xor(const RowK12& r, int m)
    {
        return RowK12 { __shfl_xor_sync(0xFFFFFFFFu, r.kl, m), __shfl_xor_sync(0xFFFFFFFFu, r.kh, m),
                        __shfl_xor_sync(0xFFFFFFFFu, r.p, m) };
    }
    __device__ __forceinline__ static RowK12 pick(bool x, const RowK12& a, const RowK12& b)
    {
        return RowK12 { x ? a.kl : b.kl, x ? a.kh : b.kh, x ? a.p : b.p };
    }
    __device__ __forceinline__ static void flip(RowK12& r, uint32_t m)
    {
        r.kl ^= m;
        r.kh ^= m;
    }
    __device__ __forceinline__ static bool marked(const RowK12& r) { return (r.kh >> 31) == 0; }
};
using RowKP = RowK12<K12_ALL>;

// Types whose equal rows are the same bits
template <class R>
struct Unique {
    static constexpr bool on = false;
};
template <>
struct Unique<RowKP> {
    static constexpr bool on = true;
};

// Types that sort with one strict compare: while a block descends its keys are
// held complemented, where the ascending compare swaps exactly the pairs that
// the descending one swaps on the plain keys (equal keys stay in both).
template <class R>
struct Flip {
    static constexpr bool on = false;
};
template <>
struct Flip<RowK12<K12_KEY>> {
    static constexpr bool on = true;
};

// Two independent 16-bit keys a row, each lane sorted on its own: an exchange
// is one packed minimum and one packed maximum for two keys (descending blocks
// are held complemented, Flip; selects by direction doubled the instructions).
struct RowU2 {
    uint32_t k;
    struct Cols {
        uint32_t* k;
    };
    static constexpr int SMEM_BYTES = 4;
    static constexpr int SWZ_BITS = 5;
    static constexpr int SLOT_BYTES = 4;
    __device__ __forceinline__ static RowU2 load(const Cols& c, size_t g)
    {
        VELO_TRACE_AT(TS_ROW_LOAD, c.k + g);
        return RowU2 { __ldcg(c.k + g) };
    }
    __device__ __forceinline__ static void store(const Cols& c, size_t g, const RowU2& r)
    {
        VELO_TRACE_AT(TS_ROW_STORE, c.k + g);
        c.k[g] = r.k;
    }
    __device__ __forceinline__ static RowU2 pad(const Cols&) { return RowU2 { ~0u }; }
    __device__ __forceinline__ static void sstore(char* sm, int, int i, const RowU2& r)
    {
        reinterpret_cast<uint32_t*>(sm)[i] = r.k;
    }
    __device__ __forceinline__ static RowU2 sload(const char* sm, int, int i)
    {
        return RowU2 { reinterpret_cast<const uint32_t*>(sm)[i] };
    }
    __device__ __forceinline__ static void sstore_b(char* sm, int, uint32_t b, const RowU2& r)
    {
        *reinterpret_cast<uint32_t*>(sm + b) = r.k;
    }
    __device__ __forceinline__ static RowU2 sload_b(const char* sm, int, uint32_t b)
    {
        return RowU2 { *reinterpret_cast<const uint32_t*>(sm + b) };
    }
    __device__ __forceinline__ static bool swap_pred(const RowU2&, const RowU2&, bool, const Cols&) { return false; }
    __device__ __forceinline__ static void cswap(RowU2& a, RowU2& b, bool)
    {
        const uint32_t lo = __vminu2(a.k, b.k);
        b.k = __vmaxu2(a.k, b.k);
        a.k = lo;
    }
    __device__ __forceinline__ static void flip(RowU2& r, uint32_t m) { r.k ^= m; }
};

// A 32-bit word as a compaction row, marked unless it is ~0 (a pair of 16-bit
// keys of rows of which one at least passes).
struct RowW {
    uint32_t k;
    struct Cols {
        uint32_t* k;
    };
    static constexpr int SMEM_BYTES = 4;
    static constexpr int SWZ_BITS = 5;
    static constexpr int SLOT_BYTES = 4;
    __device__ __forceinline__ static RowW load(const Cols& c, size_t g)
    {
        VELO_TRACE_AT(TS_ROW_LOAD, c.k + g);
        return RowW { __ldcg(c.k + g) };
    }
    __device__ __forceinline__ static void store(const Cols& c, size_t g, const RowW& r)
    {
        VELO_TRACE_AT(TS_ROW_STORE, c.k + g);
        c.k[g] = r.k;
    }
    __device__ __forceinline__ static RowW pad(const Cols&) { return RowW { ~0u }; }
    __device__ __forceinline__ static void sstore(char* sm, int, int i, const RowW& r)
    {
        reinterpret_cast<uint32_t*>(sm)[i] = r.k;
    }
    __device__ __forceinline__ static RowW sload(const char* sm, int, int i)
    {
        return RowW { reinterpret_cast<const uint32_t*>(sm)[i] };
    }
    __device__ __forceinline__ static void sstore_b(char* sm, int, uint32_t b, const RowW& r)
    {
        *reinterpret_cast<uint32_t*>(sm + b) = r.k;
    }
    __device__ __forceinline__ static RowW sload_b(const char* sm, int, uint32_t b)
    {
        return RowW { *reinterpret_cast<const uint32_t*>(sm + b) };
    }
    __device__ __forceinline__ static void cswap(RowW& a, RowW& b, bool x) { xsel(x, a.k, b.k); }
    __device__ __forceinline__ static bool marked(const RowW& r) { return r.k != ~0u; }
};

// (u64 key, u32 payload, u8 mark): compaction rows; ordered on (key, payload)
// with the mark carried, strictly.
struct RowKPM {
    uint32_t kl, kh, p, m;
    struct Cols {
        uint64_t* k;
        uint32_t* p;
        uint8_t* m;
    };
    static constexpr int SMEM_BYTES = 16; // one 16-byte slot per row (kl, kh, p, m)
    static constexpr int SWZ_BITS = 3;
    __device__ __forceinline__ static RowKPM load(const Cols& c, size_t g)
    {
        VELO_TRACE_AT(TS_ROW_LOAD, c.k + g);
        const uint64_t k = __ldcg(c.k + g);
        return RowKPM { lo32(k), hi32(k), __ldcg(c.p + g), (uint32_t)__ldcg(c.m + g) };
    }
    __device__ __forceinline__ static void store(const Cols& c, size_t g, const RowKPM& r)
    {
        VELO_TRACE_AT(TS_ROW_STORE, c.k + g);
        c.k[g] = ((uint64_t)r.kh << 32) | r.kl;
        c.p[g] = r.p;
        c.m[g] = (uint8_t)r.m;
    }
    __device__ __forceinline__ static RowKPM pad(const Cols&) { return RowKPM { ~0u, ~0u, ~0u, 0u }; }
    __device__ __forceinline__ static void sstore(char* sm, int, int i, const RowKPM& r)
    {
        reinterpret_cast<uint4*>(sm)[i] = make_uint4(r.kl, r.kh, r.p, r.m);
    }
    static constexpr int SLOT_BYTES = 16;
    __device__ __forceinline__ static void sstore_b(char* sm, int, uint32_t b, const RowKPM& r)
    {
        *reinterpret_cast<uint4*>(sm + b) = make_uint4(r.kl, r.kh, r.p, r.m);
    }
    __device__ __forceinline__ static RowKPM sload_b(const char* sm, int, uint32_t b)
    {
        const uint4 x = *reinterpret_cast<const uint4*>(sm + b);
        return RowKPM { x.x, x.y, x.z, x.w };
    }
    __device__ __forceinline__ static RowKPM sload(const char* sm, int, int i)
    {
        const uint4 x = reinterpret_cast<const uint4*>(sm)[i];
        return RowKPM { x.x, x.y, x.z, x.w };
    }
    __device__ __forceinline__ static bool swap_pred(const RowKPM& a, const RowKPM& b, bool desc, const Cols&)
    {
        const uint32_t gt = gt_mask3(a.p, a.kl, a.kh, b.p, b.kl, b.kh);
        const uint32_t lt = gt_mask3(b.p, b.kl, b.kh, a.p, a.kl, a.kh);
        return (desc ? lt : gt) != 0u;
    }
    __device__ __forceinline__ static void cswap(RowKPM& a, RowKPM& b, bool x)
    {
        // 3 M rows: ORCompact tile pass 49.2 -> 46.9 us against MadSwap
        const AddSwap m(x);
        m(a.kl, b.kl);
        m(a.kh, b.kh);
        m(a.p, b.p);
        xsel(x, a.m, b.m);
    }
    __device__ __forceinline__ static bool marked(const RowKPM& r) { return r.m != 0; }
};

// W u64 words per row (SoA).  Ordered lexicographically on the first KW words
// as KM says (masked, whole, or the high half of word 0); the mark (for
// compaction) is bit `mark_bit` of word `mark_word`, inverted when mark_inv is
// set (so an "invalid" flag can sort last).
template <int W, int KW, bool STRICT = true, int KM = KEY_MASKED>
struct RowRec {
    static_assert(KM != KEY_HI32 || KW == 1, "a 32-bit key lives in word 0");
    static constexpr int WORDS = W;
    static constexpr int KEY_WORDS = KW;
    uint64_t w[W];
    struct Cols {
        uint64_t* w[W];
        uint64_t mask[KW];
        uint64_t pad[W];
        int mark_bit;
        int mark_inv;
        int mark_word; // word holding the mark bit (0 unless set)
    };
    // smem: words 0 and 1 share a 16-byte slot (W >= 2), word 2 (W == 3) is a
    // separate 8-byte array; W == 1 uses 8-byte slots
    static constexpr int SMEM_BYTES = 8 * W + (W == 3 ? 0 : 0);
    static constexpr int SWZ_BITS = W == 1 ? 4 : 3;
    __device__ __forceinline__ static RowRec load(const Cols& c, size_t g)
    {
        VELO_TRACE_AT(TS_ROW_LOAD, c.w[0] + g);
        RowRec r;
#pragma unroll
        for (int i = 0; i < W; i++)
            r.w[i] = __ldcg(c.w[i] + g);
        return r;
    }
    __device__ __forceinline__ static void store(const Cols& c, size_t g, const RowRec& r)
    {
        VELO_TRACE_AT(TS_ROW_STORE, c.w[0] + g);
#pragma unroll
        for (int i = 0; i < W; i++)
            c.w[i][g] = r.w[i];
    }
    __device__ __forceinline__ static RowRec pad(const Cols& c)
    {
        RowRec r;
#pragma unroll
        for (int i = 0; i < W; i++)
            r.w[i] = c.pad[i];
        return r;
    }
    // slot at byte offset b = slot * SLOT_BYTES (words past the second in
    // 8-byte arrays at b / 2)
    static constexpr int SLOT_BYTES = W == 1 ? 8 : 16;
    __device__ __forceinline__ static void sstore_b(char* sm, int T, uint32_t b, const RowRec& r)
    {
        if constexpr (W == 1) {
            *reinterpret_cast<uint64_t*>(sm + b) = r.w[0];
        } else {
            *reinterpret_cast<ulonglong2*>(sm + b) = make_ulonglong2(r.w[0], r.w[1]);
#pragma unroll
            for (int x = 2; x < W; x++)
                *reinterpret_cast<uint64_t*>(sm + (size_t)16 * T + (size_t)8 * T * (x - 2) + (b >> 1)) = r.w[x];
        }
    }
    __device__ __forceinline__ static RowRec sload_b(const char* sm, int T, uint32_t b)
    {
        RowRec r;
        if constexpr (W == 1) {
            r.w[0] = *reinterpret_cast<const uint64_t*>(sm + b);
        } else {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(sm + b);
            r.w[0] = x.x;
            r.w[1] = x.y;
#pragma unroll
            for (int y = 2; y < W; y++)
                r.w[y] = *reinterpret_cast<const uint64_t*>(sm + (size_t)16 * T + (size_t)8 * T * (y - 2) + (b >> 1));
        }
        return r;
    }
    __device__ __forceinline__ static void sstore(char* sm, int T, int i, const RowRec& r)
    {
        if constexpr (W == 1) {
            reinterpret_cast<uint64_t*>(sm)[i] = r.w[0];
        } else {
            reinterpret_cast<ulonglong2*>(sm)[i] = make_ulonglong2(r.w[0], r.w[1]);
#pragma unroll
            for (int x = 2; x < W; x++)
                reinterpret_cast<uint64_t*>(sm + (size_t)16 * T + (size_t)8 * T * (x - 2))[i] = r.w[x];
        }
    }
    __device__ __forceinline__ static RowRec sload(const char* sm, int T, int i)
    {
        RowRec r;
        if constexpr (W == 1) {
            r.w[0] = reinterpret_cast<const uint64_t*>(sm)[i];
        } else {
            const ulonglong2 x = reinterpret_cast<const ulonglong2*>(sm)[i];
            r.w[0] = x.x;
            r.w[1] = x.y;
#pragma unroll
            for (int y = 2; y < W; y++)
                r.w[y] = reinterpret_cast<const uint64_t*>(sm + (size_t)16 * T + (size_t)8 * T * (y - 2))[i];
        }
        return r;
    }
    // about half of the registers on the multiply-add pipe, the rest by
    // selects (W = 1: the high half only)
    __device__ __forceinline__ static void cswap(RowRec& a, RowRec& b, bool x)
    {
        if constexpr (W == 2 && (KM == KEY_FULL || KM == KEY_HI96)) {
            // whole-word keys (the join union): 2^23-row merge 69.9 -> 62.2 us,
            // tile sort 318 -> 314 us; with a 32-bit key the tile sort's
            // three-CTA form spills (281 -> 347 us)
            const AddSwap m(x);
            m(a.w[0], b.w[0]);
            m(a.w[1], b.w[1]);
            return;
        }
        const MadSwap mad(x);
        if constexpr (W == 1) {
            uint32_t al = lo32(a.w[0]), ah = hi32(a.w[0]), bl = lo32(b.w[0]), bh = hi32(b.w[0]);
            xsel(x, al, bl);
            mad(ah, bh);
            a.w[0] = ((uint64_t)ah << 32) | al;
            b.w[0] = ((uint64_t)bh << 32) | bl;
        } else {
#pragma unroll
            for (int i = 0; i < W; i++) {
                if (2 * i < W)
                    mad(a.w[i], b.w[i]);
                else
                    xsel(x, a.w[i], b.w[i]);
            }
        }
    }
    __device__ __forceinline__ static bool swap_pred(const RowRec& a, const RowRec& b, bool desc, const Cols& c)
    {
        if constexpr (KM == KEY_HI32) {
            static_assert(STRICT, "one compare for both directions (Flip)");
            return hi32(a.w[0]) > hi32(b.w[0]);
        }
        if constexpr (KM == KEY_HI96)
            return gt_mask3(hi32(a.w[1]), lo32(a.w[0]), hi32(a.w[0]), hi32(b.w[1]), lo32(b.w[0]), hi32(b.w[0])) != 0u;
        uint64_t ka[KW], kb[KW];
#pragma unroll
        for (int x = 0; x < KW; x++) {
            ka[x] = KM == KEY_FULL ? a.w[x] : (a.w[x] & c.mask[x]);
            kb[x] = KM == KEY_FULL ? b.w[x] : (b.w[x] & c.mask[x]);
        }
        if constexpr (KW == 1)
            return STRICT ? ka[0] > kb[0] : (ka[0] > kb[0]) != desc; // (strict: Flip)
        if constexpr (STRICT) {
            const uint32_t gt = key_gt_mask<KW>(ka, kb);
            const uint32_t lt = key_gt_mask<KW>(kb, ka);
            return (desc ? lt : gt) != 0u;
        } else {
            return (key_gt_mask<KW>(ka, kb) != 0u) != desc;
        }
    }
    __device__ __forceinline__ static void flip(RowRec& r, uint32_t m)
    {
        if constexpr (KM == KEY_HI32) {
            r.w[0] ^= (uint64_t)m << 32;
        } else {
            r.w[0] ^= ((uint64_t)m << 32) | m;
            if constexpr (KM == KEY_HI96)
                r.w[1] ^= (uint64_t)m << 32;
        }
    }
    __device__ __forceinline__ static RowRec select(bool cnd, const RowRec& a, const RowRec& b)
    {
        RowRec r;
#pragma unroll
        for (int x = 0; x < W; x++)
            r.w[x] = sel(cnd, a.w[x], b.w[x]);
        return r;
    }
    __device__ __forceinline__ static bool marked_c(const RowRec& r, const Cols& c)
    {
        // AND with a per-word mask rather than selecting the word: a select
        // chain over the words is turned into a dynamically indexed load, which
        // sends the whole register tile to local memory
        const uint64_t bit = 1ull << c.mark_bit;
        uint64_t w = 0;
#pragma unroll
        for (int x = 0; x < W; x++)
            w |= r.w[x] & (c.mark_word == x ? bit : 0ull);
        return (w != 0) != (c.mark_inv != 0);
    }
};

template <>
struct Flip<RowU2> {
    static constexpr bool on = true;
};
// strict records keyed on bits of word 0 (masked, or its high half), or on word 0
// and the high half of word 1
template <int W, int KM>
struct Flip<RowRec<W, 1, true, KM>> {
    static constexpr bool on = true;
};
template <>
struct Flip<RowRec<2, 2, true, KEY_HI96>> {
    static constexpr bool on = true;
};

template <class R>
struct MarkOf {
    __device__ __forceinline__ static bool get(const R& r, const typename R::Cols&) { return R::marked(r); }
};
template <int W, int KW, bool S, int KM>
struct MarkOf<RowRec<W, KW, S, KM>> {
    __device__ __forceinline__ static bool get(const RowRec<W, KW, S, KM>& r,
                                               const typename RowRec<W, KW, S, KM>::Cols& c)
    {
        return RowRec<W, KW, S, KM>::marked_c(r, c);
    }
};

// ---------------------------------------------------------------------------
// layouts
// ---------------------------------------------------------------------------

template <int LOG_NT, int LOG_E>
struct Tile {
    static constexpr int NT = 1 << LOG_NT;
    static constexpr int E = 1 << LOG_E;
    static constexpr int LOG_T = LOG_NT + LOG_E;
    static constexpr int T = 1 << LOG_T;
    static_assert(LOG_NT >= 5, "at least one warp per CTA");

    // bank-spreading swizzle of smem slots: XOR SWZ bits taken above the
    // register window into the low bits, so the lanes of one shared-memory
    // phase (8 lanes for 16-byte slots, 16 for 8-byte slots) hit distinct
    // banks in every layout.  The source bits are never modified, so it is a
    // bijection on the tile; it is linear over XOR, so
    // swz(a | b) = swz(a) ^ swz(b) for disjoint a, b.
    template <int SWZ>
    __host__ __device__ __forceinline__ static constexpr int swz(int l)
    {
        return l ^ ((l >> (LOG_E > SWZ ? LOG_E : SWZ)) & ((1 << SWZ) - 1));
    }
};

// window start that covers bit p, going down (bitonic) or up (ORCompact)
__device__ __forceinline__ int window_down(int p, int log_e, int log_t)
{
    int s = p - log_e + 1;
    s = s < 0 ? 0 : s;
    return s > log_t - log_e ? log_t - log_e : s;
}
__device__ __forceinline__ int window_up(int p, int log_e, int log_t)
{
    int s = p;
    return s > log_t - log_e ? log_t - log_e : s;
}

} // namespace velo
