// Batched count / locate queries over a suffix-array index: a sample table of packed K-grams (every stride-th
// suffix) brackets each boundary of a query's interval, and a binary search of the suffix array inside the bracket
// finds it exactly. Results equal ref::find_one's (include/CPU_Reference.hpp:42-73).
//
// Reference behaviour followed: Sample_Table build_kernel (src/Sample_Table.cu:26-31), the bracket rules of
// table_kernel (src/Query_Engine.cu:205-279), search_kernel (:369-418) and certify_kernel (:665-686). Locate has no
// counterpart there; it lists SA[lo + k] in rank order.
#include "common.cuh"

#include <cuda.h>

#include <algorithm>
#include <atomic>

namespace
{

__global__ void table_build_kernel(const u16* __restrict__ T, const u8* __restrict__ sa40, const u64 n, const u64 stride, const u64 entries,
                                   u64* __restrict__ table)
{
    const u64 j = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(j >= entries) return;
    const u64 pos = sa40_load(sa40, j * stride);
    if(pos >= n) { table[2 * j] = 0; table[2 * j + 1] = 0; return; }
    table[2 * j] = pack4(T, pos);          // the text's zero padding pads short suffixes
    table[2 * j + 1] = pack4(T, pos + 4);
}

// Order of the suffix at `pos`, truncated to m symbols, against the pattern: -1, 0 or 1; a suffix that ends before
// m symbols while still matching is smaller (ref::cmp_suffix_pattern, include/CPU_Reference.hpp:26-36).
__device__ __forceinline__ int cmp_suffix_pattern(const u16* __restrict__ T, const u64 n, const u64 pos, const u16* __restrict__ P, const u64 m)
{
    const u64 len = (n - pos < m) ? n - pos : m;
    for(u64 i = 0; i < len; ++i)
    {
        const u16 a = T[pos + i], b = P[i];
        if(a != b) return a < b ? -1 : 1;
    }
    return len < m ? -1 : 0;
}

// The ranks that can hold the two boundaries of a query's interval, from the sample table alone.
struct Brackets { u64 lo_first, lo_last, hi_first, hi_last; };

// Up to eight symbols from address p on, most significant first, zeros behind `count` of them (1 to 8). Two 16-byte loads, the second only where the
// symbols reach into it: a piece of 16 bytes that holds a wanted symbol lies in the allocation that holds the symbol. (One symbol at a time, a
// comparison of a query's pattern with a suffix took up to sixteen loads of 32 scattered addresses each: the lines that a warp's loads touch, one a
// cycle, were three quarters of the search's time.)
__device__ __forceinline__ ulonglong2 load_symbols(const u16* p, const u32 count)
{
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    const uint4* const piece = reinterpret_cast<const uint4*>(at & ~uintptr_t(15));
    const u32 skip = u32(at >> 1) & 7u;
    const uint4 a = __ldg(piece);
    uint4 b = make_uint4(0, 0, 0, 0);
    if(skip + count > 8) b = __ldg(piece + 1);
    u32 w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    #pragma unroll
    for(int k = 0; k < 6; ++k) w[k] = (skip & 4) ? w[k + 2 < 8 ? k + 2 : 7] : w[k];
    if(skip & 4) { w[6] = 0; w[7] = 0; }
    #pragma unroll
    for(int k = 0; k < 5; ++k) w[k] = (skip & 2) ? w[k + 1] : w[k];
    u32 r[4];
    #pragma unroll
    for(int k = 0; k < 4; ++k)
    {
        const u32 v = (skip & 1) ? __funnelshift_r(w[k], w[k + 1], 16) : w[k];
        r[k] = __funnelshift_l(v, v, 16);
    }
    return make_ulonglong2((u64(r[0]) << 32) | r[1], (u64(r[2]) << 32) | r[3]);
}

// A pattern of m >= 1 symbols: its first min(m, K), packed like a table key, and the mask of those symbols.
struct Pattern
{
    u64 high = 0, low = 0, mask_high = 0, mask_low = 0, m = 0;
    __device__ __forceinline__ Pattern() {}
    __device__ __forceinline__ Pattern(const u16* P, const u64 length)
    {
        set_length(length);
        const ulonglong2 k = load_symbols(P, length < CSA_K ? u32(length) : u32(CSA_K));
        high = k.x & mask_high; low = k.y & mask_low;
    }
    __device__ __forceinline__ void set_length(const u64 length)
    {
        m = length;
        const u32 mm = m < CSA_K ? u32(m) : u32(CSA_K);
        mask_high = mm >= 4 ? ~0ull : ~0ull << (64 - 16 * mm);
        mask_low = mm <= 4 ? 0ull : (mm == 8 ? ~0ull : ~0ull << (64 - 16 * (mm - 4)));
    }
    // For patterns of at most K symbols.
    __device__ __forceinline__ bool last_is_zero() const { return ((m <= 4 ? high >> (64 - 16 * m) : low >> (128 - 16 * m)) & 0xFFFFu) == 0; }
    // The (masked) key t is smaller than the pattern's; not greater.
    __device__ __forceinline__ bool less(const ulonglong2 t) const { const u64 h = t.x & mask_high; return h < high || (h == high && (t.y & mask_low) < low); }
    __device__ __forceinline__ bool not_greater(const ulonglong2 t) const { const u64 h = t.x & mask_high; return h < high || (h == high && (t.y & mask_low) <= low); }

    // Order of the suffix at `pos`, truncated to m symbols, against the pattern, as cmp_suffix_pattern tells it. The text's zero padding may
    // only make a short suffix look equal, never greater. P: the whole pattern, read where it has more than K symbols.
    __device__ __forceinline__ int compare(const u16* __restrict__ T, const u64 n, const u64 pos, const u16* __restrict__ P) const
    {
        const ulonglong2 t = load_symbols(T + pos, m < CSA_K ? u32(m) : u32(CSA_K));
        const u64 h = t.x & mask_high, l = t.y & mask_low;
        if(h != high) return h < high ? -1 : 1;
        if(l != low) return l < low ? -1 : 1;
        for(u64 i = CSA_K; i < m; i += CSA_K)
        {
            if(pos + i >= n) return -1;
            const u32 more = m - i < CSA_K ? u32(m - i) : u32(CSA_K);
            const u64 keep_high = more >= 4 ? ~0ull : ~0ull << (64 - 16 * more), keep_low = more <= 4 ? 0ull : (more == 8 ? ~0ull : ~0ull << (64 - 16 * (more - 4)));
            const ulonglong2 x = load_symbols(T + pos + i, more), y = load_symbols(P + i, more);
            if(((x.x ^ y.x) & keep_high) != 0) return (x.x & keep_high) < (y.x & keep_high) ? -1 : 1;
            if(((x.y ^ y.y) & keep_low) != 0) return (x.y & keep_low) < (y.y & keep_low) ? -1 : 1;
        }
        return n - pos < m ? -1 : 0;
    }
};

// Entry r of a suffix array in device memory, by one 16-byte load as a rule and a second one for the quarter of the entries that cross a boundary.
__device__ __forceinline__ u64 sa40_load_wide(const u8* sa, const u64 r)
{
    const uintptr_t at = reinterpret_cast<uintptr_t>(sa) + 5 * r;
    const uint4* const piece = reinterpret_cast<const uint4*>(at & ~uintptr_t(15));
    const u32 byte = u32(at) & 15u, word = byte >> 2;
    const uint4 a = __ldg(piece);
    u32 next = 0;
    if(byte > 11) next = __ldg(reinterpret_cast<const u32*>(piece + 1));
    const u32 lo = word == 0 ? a.x : word == 1 ? a.y : word == 2 ? a.z : a.w;
    const u32 hi = word == 0 ? a.y : word == 1 ? a.z : word == 2 ? a.w : next;
    const u64 v = (u64(hi) << 32) | lo;
    return (v >> ((byte & 3) * 8)) & 0xFFFFFFFFFFull;
}

// The brackets from a = table keys (masked) smaller than the pattern's and b = those not greater, of J. Sampled rank j * stride carries
// table key j. Ranks up to (a-1) stride are smaller than the pattern; ranks from b stride on are greater.
__device__ __forceinline__ Brackets brackets_from(const u64 a, const u64 b, const u64 J, const u64 stride, const u64 ne, const Pattern& p)
{
    const u64 m = p.m;
    Brackets br;
    br.lo_first = (a == 0) ? 0 : (a - 1) * stride + 1;
    br.hi_last = (b >= J) ? ne : b * stride;
    br.lo_last = br.hi_last;
    br.hi_first = br.lo_first;
    if(m <= CSA_K)
    {
        // Every suffix whose masked key equals the pattern's matches it, except suffixes that end inside the pattern and
        // owe the equality to zero padding; there are fewer than m of them and they need the pattern to end in a zero.
        const u64 e = p.last_is_zero() ? m - 1 : 0;
        const u64 cap = a * stride + e;
        if(cap < br.lo_last) br.lo_last = cap;
        if(b > 0 && (b - 1) * stride + 1 > br.hi_first) br.hi_first = (b - 1) * stride + 1;
    }
    return br;
}

// a0, a1: the number of smaller keys lies between them; b0, b1: the number of keys not greater does.
__device__ __forceinline__ Brackets table_brackets(const csa_index& idx, const Pattern& p, const u64 a0, const u64 a1, const u64 b0, const u64 b1)
{
    const u64 stride = idx.stride;
    const u64 ne = idx.sa_entries ? idx.sa_entries : idx.n;      // entries of the suffix array (a slice of it in a sharded index)
    const u64 J = (ne + stride - 1) / stride;
    const ulonglong2* const tab = reinterpret_cast<const ulonglong2*>(idx.table);
    u64 a, b;
    {
        u64 x = a0, y = a1;
        while(x < y)
        {
            const u64 mid = x + ((y - x) >> 1);
            if(p.less(__ldg(tab + mid))) x = mid + 1; else y = mid;
        }
        a = x;
        // b lies at or shortly after a unless the pattern's K-gram is very frequent: gallop from a (1, 2, 4, ... keys ahead)
        // to the first key that is greater, then bisect what is left. Every probe is a dependent random read, and this
        // spares about twenty of them per query.
        if(x < b0) x = b0;
        y = b1;
        for(u64 step = 1; x < y; step <<= 1)
        {
            const u64 mid = (x + step - 1 < y) ? x + step - 1 : y - 1;
            if(p.not_greater(__ldg(tab + mid))) x = mid + 1; else { y = mid; break; }
        }
        while(x < y)
        {
            const u64 mid = x + ((y - x) >> 1);
            if(p.not_greater(__ldg(tab + mid))) x = mid + 1; else y = mid;
        }
        b = x;
    }
    return brackets_from(a, b, J, stride, ne, p);
}

__device__ __forceinline__ Brackets table_brackets(const csa_index& idx, const Pattern& p)
{
    const u64 ne = idx.sa_entries ? idx.sa_entries : idx.n, J = (ne + idx.stride - 1) / idx.stride;
    return table_brackets(idx, p, 0, J, 0, J);
}

// The first index of [x, y) for which `before` does not hold (y if it holds for all), by a warp: 32 probes at a time, which cut the range
// to a 33rd. before(i) is called for i in [x, y) alone.
template <typename F>
__device__ __forceinline__ u64 warp_partition_point(u64 x, u64 y, const F& before)
{
    const u32 lane = lane_id();
    while(x < y)
    {
        const u64 len = y - x;
        if(len <= 32)
        {
            const u32 held = __ballot_sync(0xFFFFFFFFu, lane < len && before(x + lane));
            return x + __popc(held);
        }
        // probes x + (k + 1) len / 33 - 1 of k = 0 .. 31: ascending, inside the range
        const u64 each = len / 33, rest = len % 33;
        auto probe = [&](const u32 k) { return x + (k + 1) * each + (k + 1) * rest / 33 - 1; };
        const u32 held = __popc(__ballot_sync(0xFFFFFFFFu, before(probe(lane) > x ? probe(lane) : x)));
        const u64 last_held = held ? probe(held - 1) : 0, first_not = held < 32 ? probe(held) : y;
        if(held < 32) y = first_not > x ? first_not : x;
        if(held) x = (last_held > x ? last_held : x) + 1;
    }
    return x;
}

// The same where the answer is likely to lie within 32 of x: that window first.
template <typename F>
__device__ __forceinline__ u64 warp_partition_point_near(u64 x, u64 y, const F& before)
{
    if(y - x > 32)
    {
        const u32 held = __popc(__ballot_sync(0xFFFFFFFFu, before(x + lane_id())));
        if(held < 32) return x + held;
        x += 32;
    }
    return warp_partition_point(x, y, before);
}

// Both boundaries of the interval by binary search inside the brackets. sa_lo(r), sa_hi(r): entry r of the suffix array in each search: of
// the array itself, or of a gathered window.
template <typename Lo, typename Hi>
__device__ __forceinline__ void search_brackets(const csa_index& idx, const Brackets& br, const Pattern& p, const u16* __restrict__ P, const Lo& sa_lo, const Hi& sa_hi,
                                                u64& lo_out, u64& hi_out)
{
    const u64 n = idx.n;
    const u16* const T = idx.text;
    u64 x = br.lo_first, y = br.lo_last;
    int found = 2;              // how the suffix at y compares, once it has been looked at
    while(x < y)
    {
        const u64 mid = x + ((y - x) >> 1);
        const int c = p.compare(T, n, sa_lo(mid), P);
        if(c < 0) x = mid + 1; else { y = mid; found = c; }
    }
    lo_out = x;
    // The first suffix that is not smaller has been looked at as a rule: the pattern does not occur, or the interval's end lies behind it (two of seven probes on average; large
    // batches take 6 to 8 % less).
    if(br.hi_first <= x && x < br.hi_last)
    {
        if(found == 1) { hi_out = x; return; }
        if(found == 0) ++x;
    }
    x = (br.hi_first > x) ? br.hi_first : x;
    y = br.hi_last;
    if(x > y) x = y;
    // most patterns occur a few times: the end of the interval is galloped to from its start, then bisected
    for(u64 step = 1; x < y; step <<= 1)
    {
        const u64 mid = (x + step - 1 < y) ? x + step - 1 : y - 1;
        if(p.compare(T, n, sa_hi(mid), P) <= 0) x = mid + 1; else { y = mid; break; }
    }
    while(x < y)
    {
        const u64 mid = x + ((y - x) >> 1);
        if(p.compare(T, n, sa_hi(mid), P) <= 0) x = mid + 1; else y = mid;
    }
    hi_out = x;
}

__device__ __forceinline__ bool is_slice(const csa_index& idx) { return idx.sa_entries != 0 && idx.sa_entries < idx.n; }

// The interval of one symbol in a whole index. A warp whose patterns are all of that length spares the loads and instructions of eight symbols (2 * 10^6 of them on 10^5
// tokens: 211 us symbol by symbol, 259 by eight, 177 this way). A function of its own, so that the search of longer ones keeps its registers.
__device__ __noinline__ void find_one_symbol(const u16* __restrict__ T, const u8* __restrict__ sa, const ulonglong2* __restrict__ tab, const u64 n, const u64 stride, const u32 c,
                                             u64* __restrict__ itv)
{
    // the first index of [x, y) with a greater symbol (`behind`), or one that is not smaller
    auto key = [&](const u64 j) { return u32(__ldg(&tab[j].x) >> 48); };
    auto symbol = [&](const u64 r) { return u32(__ldg(T + sa40_load(sa, r))); };
    auto first_from = [&](u64 x, u64 y, const auto& of) { while(x < y) { const u64 mid = x + ((y - x) >> 1); if(of(mid) < c) x = mid + 1; else y = mid; } return x; };
    auto first_behind = [&](u64 x, u64 y, const auto& of)
    {
        for(u64 step = 1; x < y; step <<= 1)
        {
            const u64 mid = (x + step - 1 < y) ? x + step - 1 : y - 1;
            if(of(mid) <= c) x = mid + 1; else { y = mid; break; }
        }
        while(x < y) { const u64 mid = x + ((y - x) >> 1); if(of(mid) <= c) x = mid + 1; else y = mid; }
        return x;
    };
    const u64 J = (n + stride - 1) / stride, a = first_from(0, J, key), b = first_behind(a, J, key);
    // every suffix whose first symbol is c matches, so the ranks between the first and the last such key do
    const u64 hi_last = b >= J ? n : b * stride, lo_last = a * stride < hi_last ? a * stride : hi_last;
    const u64 lo = first_from(a == 0 ? 0 : (a - 1) * stride + 1, lo_last, symbol);
    u64 x = b > 0 ? (b - 1) * stride + 1 : 0;
    if(lo > x) x = lo;
    if(x > hi_last) x = hi_last;
    itv[0] = lo;
    itv[1] = first_behind(x, hi_last, symbol);
}

__global__ void __launch_bounds__(128) find_kernel(const csa_index idx, const u64* __restrict__ off, const u16* __restrict__ sym, const u64 q, u64* __restrict__ itv)
{
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(i >= q) return;
    const u64 from = off[i], m = off[i + 1] - from;
    const u16* const P = sym + (from - off[0]);
    if(m == 0) { itv[2 * i] = 0; itv[2 * i + 1] = idx.sa_entries ? idx.sa_entries : idx.n; return; }
    if(__all_sync(__activemask(), m == 1 && !is_slice(idx)))
    {
        find_one_symbol(idx.text, idx.sa40, reinterpret_cast<const ulonglong2*>(idx.table), idx.n, idx.stride, P[0], itv + 2 * i);
        return;
    }
    const Pattern p(P, m);
    if(is_slice(idx))
    {
        // One slice of a sharded array: most patterns lie wholly before or wholly after it, which its first and last suffix
        // tell with two comparisons; only a pattern that falls inside the slice's range is searched for.
        const u64 e = idx.sa_entries;
        if(p.compare(idx.text, idx.n, sa40_load(idx.sa40, 0), P) > 0) { itv[2 * i] = 0; itv[2 * i + 1] = 0; return; }
        if(p.compare(idx.text, idx.n, sa40_load(idx.sa40, e - 1), P) < 0) { itv[2 * i] = e; itv[2 * i + 1] = e; return; }
    }
    const Brackets br = table_brackets(idx, p);
    u64 lo, hi;
    auto entry = [&](const u64 r) { return sa40_load_wide(idx.sa40, r); };
    search_brackets(idx, br, p, P, entry, entry, lo, hi);
    itv[2 * i] = lo;
    itv[2 * i + 1] = hi;
}

// ---- large batches: the queries by where they lie in the table ---------------------------------------------------------------
//
// A query's reads are random ones, in the table, in the array and in the text, and a batch in its own order shares none of them. So the
// queries of a large batch are first dealt into SLOTS by where they fall among as many keys of the table (a directory that a block keeps in shared
// memory): the queries of a slot then read the same upper levels of the table's bisection, one stretch of the table and one of
// the array. Nothing is sorted: the slots are counted, and a query takes the next place of its slot.
constexpr u32 SLOT_BITS = 12, SLOTS = 1u << SLOT_BITS;
constexpr int SLOT_BLOCK = 512, SLOT_ITEMS = 2, SLOT_TILE = SLOT_BLOCK * SLOT_ITEMS;
constexpr size_t SLOT_SMEM = (SLOTS + SLOTS / 16) * 8 + (SLOTS + 1) * 4;

// What a query needs on its way, in the order of the slots.
struct __align__(16) Slot_Query
{
    u64 high, low;          // Pattern
    u32 index;              // of the query in its batch
    u16 first, last;        // of the directory's keys those before `first` are smaller, those from `last` on greater
    u64 at;                 // the pattern's first symbol in the batch's, and from bit 48 on its length (LONG_PATTERN: that or more)
};
static_assert(sizeof(Slot_Query) == 32, "one sector");
constexpr u32 LONG_PATTERN = 0xFFFF;
// Blocks of 128 threads an SM that the search of dealt queries leaves registers for: more reads in flight against spills (2 * 10^6 queries of 1 to 16 symbols on
// 3 * 10^8 tokens, us a call: 8 blocks 624, 10 612, 12 626; of 2 to 4 symbols 565, 545 and 561).
constexpr int FIND_DEALT_BLOCKS = 10;

// Where a query falls in the directory, and which of its block's queries in that slot it is.
struct Slot_Place { u16 first, last; u32 rank; };

__device__ __forceinline__ u64 slot_entry(const u32 k, const u64 J) { return u64(k) * J >> SLOT_BITS; }       // J < 2^40

__global__ void __launch_bounds__(256) directory_kernel(const u64* __restrict__ table, const u64 J, u64* __restrict__ directory, u32* __restrict__ counts)
{
    const u32 k = blockIdx.x * 256 + threadIdx.x;
    if(k < SLOTS) directory[k] = table[2 * slot_entry(k, J)];       // the first four symbols
    if(k <= SLOTS) counts[k] = 0;
}

// off: the offsets of this share of the batch, off_first: the batch's first, where sym begins.
// counts[s]: queries of slot s (there is one more than directory keys). before[block][s]: those of the slot in blocks that came earlier.
__global__ void __launch_bounds__(SLOT_BLOCK) count_slots_kernel(const u64* __restrict__ directory, const u64* __restrict__ off, const u64* __restrict__ off_first, const u16* __restrict__ sym, const u64 q,
                                                                Slot_Place* __restrict__ places, u32* __restrict__ counts, u32* __restrict__ before)
{
    // A word is left free behind every sixteen keys: the probes of a bisection are a power of two apart, which without would lie in one bank (4e6 queries: 102 us, this way 70).
    extern __shared__ __align__(16) u64 dir_spread[];
    auto dir = [&](const u32 k) -> u64& { return dir_spread[k + (k >> 4)]; };
    u32* const cnt = reinterpret_cast<u32*>(dir_spread + SLOTS + SLOTS / 16);
    for(u32 k = threadIdx.x; k < SLOTS; k += SLOT_BLOCK) { dir(k) = directory[k]; cnt[k] = 0; }
    if(threadIdx.x == 0) cnt[SLOTS] = 0;
    __syncthreads();
    const u64 off0 = *off_first;
    for(u64 tile = blockIdx.x; tile * SLOT_TILE < q; tile += gridDim.x)
    {
        Pattern ps[SLOT_ITEMS];             // their reads side by side
        #pragma unroll
        for(int k = 0; k < SLOT_ITEMS; ++k)
        {
            const u64 i = tile * SLOT_TILE + k * SLOT_BLOCK + threadIdx.x;
            if(i >= q) continue;
            const u64 from = off[i], m = off[i + 1] - from;
            if(m) ps[k] = Pattern(sym + (from - off0), m);
        }
        #pragma unroll
        for(int k = 0; k < SLOT_ITEMS; ++k)
        {
            const u64 i = tile * SLOT_TILE + k * SLOT_BLOCK + threadIdx.x;
            if(i >= q) continue;
            const Pattern& p = ps[k];
            u32 x = 0, z = 0;
            if(p.m)
            {
                #pragma unroll
                for(u32 step = SLOTS / 2; step; step >>= 1) if((dir(x + step - 1) & p.mask_high) < p.high) x += step;
                if(x == SLOTS - 1 && (dir(x) & p.mask_high) < p.high) ++x;
                z = x;
                u32 y = SLOTS;
                for(u32 step = 1; z < y; step <<= 1)
                {
                    const u32 mid = min(z + step - 1, y - 1);
                    if((dir(mid) & p.mask_high) <= p.high) z = mid + 1; else { y = mid; break; }
                }
                while(z < y)
                {
                    const u32 mid = (z + y) >> 1;
                    if((dir(mid) & p.mask_high) <= p.high) z = mid + 1; else y = mid;
                }
            }
            places[i] = Slot_Place{u16(x), u16(z), atomicAdd(&cnt[x], 1u)};
        }
    }
    __syncthreads();
    for(u32 k = threadIdx.x; k <= SLOTS; k += SLOT_BLOCK)
    {
        const u32 c = cnt[k];
        if(c) before[u64(blockIdx.x) * (SLOTS + 1) + k] = atomicAdd(&counts[k], c);
    }
}

// The queries in the order of their slots; the same blocks take the same queries as in the kernel above.
__global__ void __launch_bounds__(SLOT_BLOCK) deal_slots_kernel(const u64* __restrict__ off, const u64* __restrict__ off_first, const u16* __restrict__ sym, const u64 q, const Slot_Place* __restrict__ places,
                                                               const u32* __restrict__ counts, const u32* __restrict__ before, Slot_Query* __restrict__ dealt)
{
    __shared__ u32 first_of[SLOTS + 1];         // where the block's queries of a slot start
    __shared__ u32 warp_tot[SLOT_BLOCK / 32];
    constexpr u32 PER = (SLOTS + SLOT_BLOCK) / SLOT_BLOCK;
    const u32 k0 = threadIdx.x * PER;
    u32 c[PER], sum = 0;
    #pragma unroll
    for(u32 k = 0; k < PER; ++k) { c[k] = k0 + k <= SLOTS ? counts[k0 + k] : 0; sum += c[k]; }
    u32 inc = sum;
    #pragma unroll
    for(int o = 1; o < 32; o <<= 1) { const u32 t = __shfl_up_sync(0xFFFFFFFFu, inc, o); if(int(lane_id()) >= o) inc += t; }
    if(lane_id() == 31) warp_tot[threadIdx.x >> 5] = inc;
    __syncthreads();
    u32 run = inc - sum;
    for(u32 w = 0; w < (threadIdx.x >> 5); ++w) run += warp_tot[w];
    #pragma unroll
    for(u32 k = 0; k < PER; ++k)
        if(k0 + k <= SLOTS) { first_of[k0 + k] = run + before[u64(blockIdx.x) * (SLOTS + 1) + k0 + k]; run += c[k]; }       // a slot without queries of this block: not used
    __syncthreads();
    const u64 off0 = *off_first;
    for(u64 tile = blockIdx.x; tile * SLOT_TILE < q; tile += gridDim.x)
        #pragma unroll
        for(int k = 0; k < SLOT_ITEMS; ++k)
        {
            const u64 i = tile * SLOT_TILE + k * SLOT_BLOCK + threadIdx.x;
            if(i >= q) continue;
            const Slot_Place pl = places[i];
            const u64 from = off[i], m = off[i + 1] - from;
            Pattern p;
            if(m) p = Pattern(sym + (from - off0), m);
            const u64 at = (from - off0) | (m < LONG_PATTERN ? m : u64(LONG_PATTERN)) << 48;
            uint4* const out = reinterpret_cast<uint4*>(dealt + first_of[pl.first] + pl.rank);
            out[0] = make_uint4(u32(p.high), u32(p.high >> 32), u32(p.low), u32(p.low >> 32));
            out[1] = make_uint4(u32(i), u32(pl.first) | u32(pl.last) << 16, u32(at), u32(at >> 32));
        }
}

__global__ void __launch_bounds__(128, FIND_DEALT_BLOCKS) find_dealt_kernel(const csa_index idx, const u64* __restrict__ off, const u16* __restrict__ sym, const Slot_Query* __restrict__ dealt,
                                                                           const u64 q, u64* __restrict__ itv)
{
    const u64 t = u64(blockIdx.x) * 128 + threadIdx.x;
    if(t >= q) return;
    const uint4 r0 = __ldcs(reinterpret_cast<const uint4*>(dealt + t)), r1 = __ldcs(reinterpret_cast<const uint4*>(dealt + t) + 1);
    const u64 i = r1.x, at = (u64(r1.w) << 32) | r1.z;
    u64 m = at >> 48;
    if(m == LONG_PATTERN) m = off[i + 1] - off[i];
    ulonglong2 answer = make_ulonglong2(0, idx.n);
    if(m)
    {
        const u16* const P = sym + (at & ((u64(1) << 48) - 1));
        Pattern p;
        p.set_length(m);
        p.high = (u64(r0.y) << 32) | r0.x; p.low = (u64(r0.w) << 32) | r0.z;
        const u64 J = (idx.n + idx.stride - 1) / idx.stride;
        const u32 first = r1.y & 0xFFFFu, last = r1.y >> 16;
        const u64 from = first ? slot_entry(first - 1, J) + 1 : 0, to = last < SLOTS ? slot_entry(last, J) : J;
        // the directory holds four symbols of a key: of a shorter pattern it tells all
        const u64 a1 = p.mask_low ? to : (first < SLOTS ? slot_entry(first, J) : J), b0 = p.mask_low || last == 0 ? from : slot_entry(last - 1, J) + 1;
        const Brackets br = table_brackets(idx, p, from, a1, b0, to);
        auto entry = [&](const u64 r) { return sa40_load_wide(idx.sa40, r); };
        search_brackets(idx, br, p, P, entry, entry, answer.x, answer.y);
    }
    reinterpret_cast<ulonglong2*>(itv)[i] = answer;
}

// A warp per query, for batches that do not fill the device with a thread per query: what bounds those is a chain of 25 to 40 dependent
// random reads, which 32 probes at a time make four to five times shorter.
__global__ void __launch_bounds__(128) find_by_warp_kernel(const csa_index idx, const u64* __restrict__ off, const u16* __restrict__ sym, const u64 q, u64* __restrict__ itv)
{
    const u64 i = u64(blockIdx.x) * (blockDim.x / 32) + (threadIdx.x >> 5);
    if(i >= q) return;
    const u64 first = off[0], from = off[i], m = off[i + 1] - from;
    const u16* const P = sym + (from - first);
    const u64 ne = idx.sa_entries ? idx.sa_entries : idx.n, n = idx.n;
    u64 lo = 0, hi = 0;
    if(m == 0) hi = ne;
    else
    {
        const Pattern p(P, m);
        if(is_slice(idx) && p.compare(idx.text, n, sa40_load(idx.sa40, 0), P) > 0) {}      // a slice behind the pattern
        else if(is_slice(idx) && p.compare(idx.text, n, sa40_load(idx.sa40, ne - 1), P) < 0) { lo = ne; hi = ne; }
        else
        {
            const u64 J = (ne + idx.stride - 1) / idx.stride;
            const ulonglong2* const tab = reinterpret_cast<const ulonglong2*>(idx.table);
            const u64 a = warp_partition_point(0, J, [&](const u64 j) { return p.less(tab[j]); });
            const u64 b = warp_partition_point_near(a, J, [&](const u64 j) { return p.not_greater(tab[j]); });
            const Brackets br = brackets_from(a, b, J, idx.stride, ne, p);
            lo = warp_partition_point(br.lo_first, br.lo_last, [&](const u64 r) { return p.compare(idx.text, n, sa40_load(idx.sa40, r), P) < 0; });
            u64 x = br.hi_first > lo ? br.hi_first : lo;
            if(x > br.hi_last) x = br.hi_last;
            hi = warp_partition_point_near(x, br.hi_last, [&](const u64 r) { return p.compare(idx.text, n, sa40_load(idx.sa40, r), P) <= 0; });
        }
    }
    if(lane_id() == 0) { itv[2 * i] = lo; itv[2 * i + 1] = hi; }
}

// Batches up to here take a warp per query. Counting on 2e8 suffixes, a call with a thread and with a warp per query: 50 queries 54 and
// 38 us, 1000 65 and 40, 8000 63 and 44, 16000 61 and 61, 64000 77 and 125 us (on 2^24 suffixes 61 and 41 at 8000, 64 and 53 at 16000).
constexpr u64 WARP_QUERIES = 8192;

// ---- the same search when the suffix array lies in pinned host memory -------------------------------------------------
// Every probe of the array would be a PCIe round trip, so the entries of both brackets are first gathered into device
// memory, one warp per query with 16-byte loads (the reference's gather_kernel, src/Query_Engine.cu:334-354, does the same
// for its pinned plan), and the binary searches then run on the gathered windows. A bracket wider than WINDOW_ENTRIES
// (a long pattern whose K-gram prefix is very frequent) is searched in place.
constexpr u32 WINDOW_ENTRIES = 64;
constexpr u32 WINDOW_BYTES = 352;       // 5 * (WINDOW_ENTRIES + 1) entries' bytes + alignment slack + the load overrun, in 16-byte pieces

__global__ void brackets_kernel(const csa_index idx, const u64* __restrict__ off, const u16* __restrict__ sym, const u64 q, Brackets* __restrict__ out)
{
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(i >= q) return;
    const u64 m = off[i + 1] - off[i];
    Brackets br{0, 0, 0, 0};
    if(m > 0) br = table_brackets(idx, Pattern(sym + (off[i] - off[0]), m));
    out[i] = br;
}

__device__ __forceinline__ bool window_fits(u64 first, u64 last) { return last - first <= WINDOW_ENTRIES; }

__global__ void gather_windows_kernel(const u8* __restrict__ sa40, const Brackets* __restrict__ br, const u64 q, u8* __restrict__ win)
{
    const u64 w = (u64(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if(w >= q) return;
    const Brackets b = br[w];
    #pragma unroll
    for(int side = 0; side < 2; ++side)
    {
        const u64 first = side ? b.hi_first : b.lo_first, last = side ? b.hi_last : b.lo_last;
        if(last < first || !window_fits(first, last)) continue;
        if(side == 1 && b.hi_first == b.lo_first && b.hi_last == b.lo_last) continue;     // one window serves both searches (patterns longer than K)
        const u64 byte0 = (5 * first) & ~u64(15), byte1 = 5 * last + 5 + 4;       // entry `last` may be probed; a load reads 8 bytes
        const u32 pieces = u32((byte1 - byte0 + 15) >> 4);
        const uint4* src = reinterpret_cast<const uint4*>(sa40 + byte0);
        uint4* dst = reinterpret_cast<uint4*>(win + (2 * w + side) * WINDOW_BYTES);
        if(lane_id() < pieces && lane_id() < WINDOW_BYTES / 16) dst[lane_id()] = src[lane_id()];
    }
}

__global__ void search_windows_kernel(const csa_index idx, const u64* __restrict__ off, const u16* __restrict__ sym, const u64 q,
                                      const Brackets* __restrict__ brs, const u8* __restrict__ win, u64* __restrict__ itv)
{
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(i >= q) return;
    const u64 m = off[i + 1] - off[i];
    if(m == 0) { itv[2 * i] = 0; itv[2 * i + 1] = idx.sa_entries ? idx.sa_entries : idx.n; return; }
    const Brackets br = brs[i];
    // A window holds the array's bytes from (5 first) & ~15 on; shifting its base back by that much lets rank r address it.
    const u8* sa_lo = idx.sa40;
    const u8* sa_hi = idx.sa40;
    if(br.lo_last >= br.lo_first && window_fits(br.lo_first, br.lo_last)) sa_lo = win + (2 * i) * WINDOW_BYTES - ((5 * br.lo_first) & ~u64(15));
    if(br.hi_last >= br.hi_first && window_fits(br.hi_first, br.hi_last))
    {
        const bool shared = br.hi_first == br.lo_first && br.hi_last == br.lo_last;
        sa_hi = win + (2 * i + (shared ? 0 : 1)) * WINDOW_BYTES - ((5 * br.hi_first) & ~u64(15));
    }
    u64 lo, hi;
    const u16* const P = sym + (off[i] - off[0]);
    search_brackets(idx, br, Pattern(P, m), P, [&](const u64 r) { return sa40_load(sa_lo, r); }, [&](const u64 r) { return sa40_load(sa_hi, r); }, lo, hi);
    itv[2 * i] = lo;
    itv[2 * i + 1] = hi;
}

// Eight lanes per query (most match once or a few times, and half of a batch may not match at all): row i of pos receives SA[lo + k],
// k < min(max_pos, hi - lo). (A warp per query: 126 us for 10^6 queries of up to 20 positions, this way 48 us.)
constexpr u32 LOCATE_LANES = 8;

__global__ void __launch_bounds__(256) locate_rows_kernel(const u8* __restrict__ sa40, const u64* __restrict__ itv, const u64 q, const u32 max_pos, u64* __restrict__ pos,
                                                         u32* __restrict__ cnt)
{
    const u64 w = (u64(blockIdx.x) * 256 + threadIdx.x) / LOCATE_LANES;
    if(w >= q) return;
    const u64 lo = itv[2 * w], hi = itv[2 * w + 1];
    const u32 c = (hi - lo < max_pos) ? u32(hi - lo) : max_pos, lane = threadIdx.x % LOCATE_LANES;
    if(lane == 0) cnt[w] = c;
    for(u32 k = lane; k < c; k += LOCATE_LANES) pos[w * max_pos + k] = sa40_load(sa40, lo + k);
}

// The same into one packed array: query i's positions start at pos_off[i].
__global__ void __launch_bounds__(256) locate_packed_kernel(const u8* __restrict__ sa40, const u64* __restrict__ itv, const u64 q, const u32 max_pos,
                                                           const u64* __restrict__ pos_off, u64* __restrict__ pos)
{
    const u64 w = (u64(blockIdx.x) * 256 + threadIdx.x) / LOCATE_LANES;
    if(w >= q) return;
    const u64 lo = itv[2 * w], hi = itv[2 * w + 1];
    const u32 c = (hi - lo < max_pos) ? u32(hi - lo) : max_pos;
    const u64 o = pos_off[w];
    for(u32 k = threadIdx.x % LOCATE_LANES; k < c; k += LOCATE_LANES) pos[o + k] = sa40_load(sa40, lo + k);
}

// Sharded locate: the columns of a global interval's row that fall into this slice of the suffix array.
__global__ void locate_window_kernel(const u8* __restrict__ sa40, const u64 sa_first, const u64 sa_entries, const u64* __restrict__ itv, const u64 q,
                                     const u32 max_pos, u64* __restrict__ pos)
{
    const u64 w = (u64(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if(w >= q) return;
    const u64 lo = itv[2 * w], hi = itv[2 * w + 1];
    const u64 c = (hi - lo < max_pos) ? hi - lo : max_pos;
    for(u64 k = lane_id(); k < c; k += 32)
    {
        const u64 r = lo + k;
        if(r >= sa_first && r < sa_first + sa_entries) pos[w * max_pos + k] = sa40_load(sa40, r - sa_first);
    }
}

// Sharded locate into ONE packed array: the entries of a global interval's first max_pos ranks that fall into this slice go to
// pos[pos_off[i] + k] (rank lo + k); the other entries are left as they are, so packed arrays that all shards write into, starting
// from zeros, add up to the packed positions of the whole index.
__global__ void locate_window_packed_kernel(const u8* __restrict__ sa40, const u64 sa_first, const u64 sa_entries, const u64* __restrict__ itv, const u64 q,
                                            const u32 max_pos, const u64* __restrict__ pos_off, u64* __restrict__ pos)
{
    const u64 w = (u64(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if(w >= q) return;
    const u64 lo = itv[2 * w], hi = itv[2 * w + 1];
    const u64 c = (hi - lo < max_pos) ? hi - lo : max_pos;
    if(c == 0 || lo + c <= sa_first || lo >= sa_first + sa_entries) return;
    const u64 o = pos_off[w];
    for(u64 k = lane_id(); k < c; k += 32)
    {
        const u64 r = lo + k;
        if(r >= sa_first && r < sa_first + sa_entries) pos[o + k] = sa40_load(sa40, r - sa_first);
    }
}

__global__ void counts_kernel(const u64* __restrict__ itv, const u64 q, const u32 max_pos, u32* __restrict__ cnt)
{
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(i >= q) return;
    const u64 d = itv[2 * i + 1] - itv[2 * i];
    cnt[i] = u32(d < max_pos ? d : max_pos);
}

// Exclusive prefix sums of 32-bit counts into 64-bit offsets (off[count] = total), in three steps without waits:
// block sums, a one-block scan of them, and the per-block scans.
constexpr int SCAN_BLOCK = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

__global__ void __launch_bounds__(SCAN_BLOCK) scan_sums_kernel(const u32* __restrict__ in, const u64 count, u64* __restrict__ sums)
{
    __shared__ u64 s[SCAN_BLOCK / 32];
    u64 v = 0;
    const u64 first = u64(blockIdx.x) * SCAN_TILE + u64(threadIdx.x) * SCAN_ITEMS;
    for(int i = 0; i < SCAN_ITEMS; ++i) if(first + i < count) v += in[first + i];
    for(int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if(lane_id() == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if(threadIdx.x == 0) { u64 t = 0; for(int w = 0; w < SCAN_BLOCK / 32; ++w) t += s[w]; sums[blockIdx.x] = t; }
}

__global__ void __launch_bounds__(1024) scan_carry_kernel(u64* __restrict__ sums, const u64 tiles, u64* __restrict__ total)
{
    __shared__ u64 s[32];
    __shared__ u64 carry;
    if(threadIdx.x == 0) carry = 0;
    __syncthreads();
    for(u64 base = 0; base < tiles; base += 1024)
    {
        const u64 t = base + threadIdx.x;
        const u64 v = (t < tiles) ? sums[t] : 0;
        u64 inc = v;
        for(int o = 1; o < 32; o <<= 1) { const u64 u = __shfl_up_sync(0xFFFFFFFFu, inc, o); if(int(lane_id()) >= o) inc += u; }
        if(lane_id() == 31) s[threadIdx.x >> 5] = inc;
        __syncthreads();
        u64 pre = carry;
        for(u32 w = 0; w < (threadIdx.x >> 5); ++w) pre += s[w];
        __syncthreads();
        if(t < tiles) sums[t] = pre + inc - v;
        if(threadIdx.x == 1023) carry = pre + inc;
        __syncthreads();
    }
    if(threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(SCAN_BLOCK) scan_apply_kernel(const u32* __restrict__ in, const u64 count, const u64* __restrict__ sums,
                                                               const u64* __restrict__ total, u64* __restrict__ out)
{
    __shared__ u64 s[SCAN_BLOCK / 32];
    const u64 first = u64(blockIdx.x) * SCAN_TILE + u64(threadIdx.x) * SCAN_ITEMS;
    u32 v[SCAN_ITEMS];
    u64 mine = 0;
    for(int i = 0; i < SCAN_ITEMS; ++i) { v[i] = (first + i < count) ? in[first + i] : 0; mine += v[i]; }
    u64 inc = mine;
    for(int o = 1; o < 32; o <<= 1) { const u64 u = __shfl_up_sync(0xFFFFFFFFu, inc, o); if(int(lane_id()) >= o) inc += u; }
    if(lane_id() == 31) s[threadIdx.x >> 5] = inc;
    __syncthreads();
    u64 run = sums[blockIdx.x] + inc - mine;
    for(u32 w = 0; w < (threadIdx.x >> 5); ++w) run += s[w];
    for(int i = 0; i < SCAN_ITEMS; ++i)
    {
        if(first + i < count) out[first + i] = run;
        run += v[i];
    }
    if(blockIdx.x == 0 && threadIdx.x == 0) out[count] = *total;
}

__global__ void certify_kernel(const csa_index idx, const u64* __restrict__ off, const u16* __restrict__ sym, const u64 q, const u64* __restrict__ itv,
                               u64* __restrict__ result)
{
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(i >= q) return;
    const u64 n = idx.n, m = off[i + 1] - off[i], lo = itv[2 * i], hi = itv[2 * i + 1];
    const u16* const P = sym + (off[i] - off[0]);
    bool ok = true;
    if(lo > hi || hi > n) ok = false;
    else if(m == 0) ok = (lo == 0 && hi == n);
    else
    {
        if(lo > 0 && cmp_suffix_pattern(idx.text, n, sa40_load(idx.sa40, lo - 1), P, m) >= 0) ok = false;
        if(ok && lo < hi && (cmp_suffix_pattern(idx.text, n, sa40_load(idx.sa40, lo), P, m) != 0
                             || cmp_suffix_pattern(idx.text, n, sa40_load(idx.sa40, hi - 1), P, m) != 0)) ok = false;
        if(ok && hi < n && cmp_suffix_pattern(idx.text, n, sa40_load(idx.sa40, hi), P, m) <= 0) ok = false;
    }
    if(!ok)
    {
        atomicAdd(&result[0], 1ull);
        atomicMin(&result[1], i);
    }
}

int check_index(csa_ctx* ctx, const csa_index* index)
{
    if(!ctx || !index || !index->text || !index->sa40 || !index->table || index->n == 0 || index->stride == 0)
        return csa_fail(ctx, CSA_E_INVALID, "query: incomplete index");
    if(reinterpret_cast<uintptr_t>(index->sa40) & 3) return csa_fail(ctx, CSA_E_INVALID, "query: the suffix array must be 4-byte aligned");
    if(reinterpret_cast<uintptr_t>(index->table) & 15) return csa_fail(ctx, CSA_E_INVALID, "query: the sample table must be 16-byte aligned");
    return CSA_OK;
}

int exclusive_sum(csa_ctx* ctx, const u32* in, u64 count, u64* out, u64* sums_scratch, u64* total_dev)
{
    const u64 tiles = div_up(count, SCAN_TILE);
    if(tiles == 0) { CSA_CUDA(ctx, cudaMemsetAsync(out, 0, 8, ctx->stream)); CSA_CUDA(ctx, cudaMemsetAsync(total_dev, 0, 8, ctx->stream)); return CSA_OK; }
    scan_sums_kernel<<<unsigned(tiles), SCAN_BLOCK, 0, ctx->stream>>>(in, count, sums_scratch);
    CSA_LAUNCH_CHECK(ctx);
    scan_carry_kernel<<<1, 1024, 0, ctx->stream>>>(sums_scratch, tiles, total_dev);
    CSA_LAUNCH_CHECK(ctx);
    scan_apply_kernel<<<unsigned(tiles), SCAN_BLOCK, 0, ctx->stream>>>(in, count, sums_scratch, total_dev, out);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

}   // namespace

extern "C" int csa_table_build(csa_ctx* ctx, const uint16_t* text, uint64_t n, const uint8_t* sa40, uint64_t stride, uint64_t* table)
{
    if(!ctx || !text || !sa40 || !table || n == 0 || stride == 0) return csa_fail(ctx, CSA_E_INVALID, "csa_table_build: bad argument");
    if(reinterpret_cast<uintptr_t>(sa40) & 3) return csa_fail(ctx, CSA_E_INVALID, "csa_table_build: the suffix array must be 4-byte aligned");
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    const u64 entries = div_up(n, stride);
    table_build_kernel<<<unsigned(div_up(entries, 256)), 256, 0, ctx->stream>>>(text, sa40, n, stride, entries, reinterpret_cast<u64*>(table));
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

extern "C" int csa_table_build_slice(csa_ctx* ctx, const uint16_t* text, uint64_t n, const uint8_t* sa40_slice, uint64_t sa_entries, uint64_t stride,
                                     uint64_t* table)
{
    if(!ctx || !text || !sa40_slice || !table || n == 0 || stride == 0 || sa_entries > n) return csa_fail(ctx, CSA_E_INVALID, "csa_table_build_slice: bad argument");
    if(reinterpret_cast<uintptr_t>(sa40_slice) & 3) return csa_fail(ctx, CSA_E_INVALID, "csa_table_build_slice: the slice must start 4-byte aligned");
    if(sa_entries == 0) return CSA_OK;
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    const u64 entries = div_up(sa_entries, stride);
    table_build_kernel<<<unsigned(div_up(entries, 256)), 256, 0, ctx->stream>>>(text, sa40_slice, n, stride, entries, reinterpret_cast<u64*>(table));
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

extern "C" int csa_locate_window(csa_ctx* ctx, const csa_index* index, const uint64_t* itv, uint64_t q, uint32_t max_pos, uint64_t* pos)
{
    CSA_TRY(check_index(ctx, index));
    if(q == 0) return CSA_OK;
    if(!itv || !pos || max_pos == 0) return csa_fail(ctx, CSA_E_INVALID, "csa_locate_window: bad argument");
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    const u64 ne = index->sa_entries ? index->sa_entries : index->n;
    locate_window_kernel<<<unsigned(div_up(q * 32, 256)), 256, 0, ctx->stream>>>(index->sa40, index->sa_first, ne, reinterpret_cast<const u64*>(itv), q, max_pos,
                                                                                 reinterpret_cast<u64*>(pos));
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

extern "C" int csa_locate_window_packed(csa_ctx* ctx, const csa_index* index, const uint64_t* itv, uint64_t q, uint32_t max_pos, uint32_t* cnt, uint64_t* pos_off,
                                        uint64_t* pos, uint64_t* total)
{
    CSA_TRY(check_index(ctx, index));
    if(q == 0) return CSA_OK;
    if(!itv || !cnt || !pos_off || !pos || !total || max_pos == 0) return csa_fail(ctx, CSA_E_INVALID, "csa_locate_window_packed: bad argument");
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    void* ws = nullptr;
    CSA_TRY(csa_aux(ctx, align_up256((div_up(q, SCAN_TILE) + 1) * 8), &ws));
    counts_kernel<<<unsigned(div_up(q, 256)), 256, 0, ctx->stream>>>(reinterpret_cast<const u64*>(itv), q, max_pos, cnt);
    CSA_LAUNCH_CHECK(ctx);
    CSA_TRY(exclusive_sum(ctx, cnt, q, reinterpret_cast<u64*>(pos_off), static_cast<u64*>(ws), reinterpret_cast<u64*>(total)));
    const u64 ne = index->sa_entries ? index->sa_entries : index->n;
    locate_window_packed_kernel<<<unsigned(div_up(q * 32, 256)), 256, 0, ctx->stream>>>(index->sa40, index->sa_first, ne, reinterpret_cast<const u64*>(itv), q, max_pos,
                                                                                        reinterpret_cast<const u64*>(pos_off), reinterpret_cast<u64*>(pos));
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

namespace
{

// A batch by slots, 2^22 queries at a time (the scratch is bounded: 180 MB). done stays false where nothing was queued: no room for the scratch, a
// stream that is being captured (an allocation is not allowed there), a slice of an index, or a batch or a table below the sizes from which on it
// pays: dealing costs what the searches spare until batches share much of a table beyond L2. us a batch, dealt and in its own order: 5e8 tokens (stride 32)
// 2^18 queries 169 and 157, 2^19 250 and 277, 2e6 645 and 797; 2e8 tokens 2^19 222 and 232, 2e6 568 and 661; 5e7 tokens (1.6e6 keys) 2^19 182 and 166, 2e6 456 and 462.
constexpr u64 DEAL_MIN_QUERIES = u64(1) << 19, DEAL_MIN_KEYS = u64(1) << 22, DEAL_CHUNK = u64(1) << 22;

int find_dealt(csa_ctx* ctx, const csa_index& index, const u64* off, const u16* sym, const u64 q, u64* itv, bool& done)
{
    const u64 J = div_up(index.n, index.stride);
    if((index.sa_entries != 0 && index.sa_entries < index.n) || J < DEAL_MIN_KEYS || J >= (u64(1) << 40)) return CSA_OK;
    if(reinterpret_cast<uintptr_t>(itv) & 15) return CSA_OK;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if(cudaStreamIsCapturing(ctx->stream, &capturing) != cudaSuccess) { cudaGetLastError(); return CSA_OK; }
    if(capturing != cudaStreamCaptureStatusNone) return CSA_OK;
    const u64 per = std::min(q, DEAL_CHUNK);
    const unsigned most_blocks = unsigned(std::min<u64>(div_up(per, SLOT_TILE), 148 * 4));
    const size_t b_dealt = align_up256(per * sizeof(Slot_Query)), b_places = align_up256(per * sizeof(Slot_Place)), b_dir = align_up256(SLOTS * 8), b_counts = align_up256((SLOTS + 1) * 4),
                 b_before = align_up256(size_t(most_blocks) * (SLOTS + 1) * 4);
    void* aux = nullptr;
    const std::string err = ctx->err;
    if(const int rc = csa_aux(ctx, b_dealt + b_places + b_dir + b_counts + b_before, &aux)) { if(rc != CSA_E_NOMEM) return rc; ctx->err = err; return CSA_OK; }
    u8* at = static_cast<u8*>(aux);
    Slot_Query* const dealt = reinterpret_cast<Slot_Query*>(at); at += b_dealt;
    Slot_Place* const places = reinterpret_cast<Slot_Place*>(at); at += b_places;
    u64* const directory = reinterpret_cast<u64*>(at); at += b_dir;
    u32* const counts = reinterpret_cast<u32*>(at); at += b_counts;
    u32* const before = reinterpret_cast<u32*>(at);
    static std::atomic<bool> configured[64];
    if(!configured[ctx->device & 63])
    {
        CSA_CUDA(ctx, cudaFuncSetAttribute(count_slots_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SLOT_SMEM)));
        configured[ctx->device & 63] = true;
    }
    for(u64 first = 0; first < q; first += per)
    {
        const u64 c = std::min(per, q - first);
        const unsigned blocks = unsigned(std::min<u64>(div_up(c, SLOT_TILE), most_blocks));
        directory_kernel<<<unsigned(div_up(SLOTS + 1, 256)), 256, 0, ctx->stream>>>(reinterpret_cast<const u64*>(index.table), J, directory, counts);
        CSA_LAUNCH_CHECK(ctx);
        count_slots_kernel<<<blocks, SLOT_BLOCK, SLOT_SMEM, ctx->stream>>>(directory, off + first, off, sym, c, places, counts, before);
        CSA_LAUNCH_CHECK(ctx);
        deal_slots_kernel<<<blocks, SLOT_BLOCK, 0, ctx->stream>>>(off + first, off, sym, c, places, counts, before, dealt);
        CSA_LAUNCH_CHECK(ctx);
        find_dealt_kernel<<<unsigned(div_up(c, 128)), 128, 0, ctx->stream>>>(index, off + first, sym, dealt, c, itv + 2 * first);
        CSA_LAUNCH_CHECK(ctx);
    }
    done = true;
    return CSA_OK;
}

// may_deal: the context's second buffer is free for the batch's scratch (the lanes of a host batch share it).
int find_batch(csa_ctx* ctx, const csa_index* index, const uint64_t* off, const uint16_t* sym, uint64_t q, uint64_t* itv, const bool may_deal)
{
    CSA_TRY(check_index(ctx, index));
    if(q == 0) return CSA_OK;
    if(!off || !itv) return csa_fail(ctx, CSA_E_INVALID, "csa_find: null buffer");
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaPointerAttributes attr;
    const bool sa_on_host = cudaPointerGetAttributes(&attr, index->sa40) == cudaSuccess && attr.type == cudaMemoryTypeHost;
    cudaGetLastError();
    if(!sa_on_host)
    {
        if(q >= DEAL_MIN_QUERIES && may_deal)
        {
            bool done = false;
            CSA_TRY(find_dealt(ctx, *index, reinterpret_cast<const u64*>(off), sym, q, reinterpret_cast<u64*>(itv), done));
            if(done) return CSA_OK;
        }
        if(q <= WARP_QUERIES) find_by_warp_kernel<<<unsigned(div_up(q, 4)), 128, 0, ctx->stream>>>(*index, reinterpret_cast<const u64*>(off), sym, q, reinterpret_cast<u64*>(itv));
        else find_kernel<<<unsigned(div_up(q, 128)), 128, 0, ctx->stream>>>(*index, reinterpret_cast<const u64*>(off), sym, q, reinterpret_cast<u64*>(itv));
        CSA_LAUNCH_CHECK(ctx);
        return CSA_OK;
    }
    // Suffix array in pinned host memory: brackets from the table, the brackets' entries gathered over PCIe, search on the
    // device. Batches of 2^20 queries bound the window buffer (about 0.8 GB).
    constexpr u64 BATCH = u64(1) << 20;
    const u64 per = (q < BATCH ? q : BATCH);
    void* aux = nullptr;
    CSA_TRY(csa_aux(ctx, align_up256(per * sizeof(Brackets)) + align_up256(per * 2 * WINDOW_BYTES + 256), &aux));
    Brackets* brs = static_cast<Brackets*>(aux);
    u8* win = static_cast<u8*>(aux) + align_up256(per * sizeof(Brackets));
    for(u64 first = 0; first < q; first += BATCH)
    {
        const u64 c = (q - first < BATCH ? q - first : BATCH);
        const u64* o = reinterpret_cast<const u64*>(off) + first;
        // The kernels address pattern i at sym + (off[i] - off[0]) of the offsets they are given, so a later batch gets the
        // symbol pointer moved on by the symbols that precede it.
        const u16* sy = sym;
        if(first > 0)
        {
            u64 begin[2] = {0, 0};
            CSA_CUDA(ctx, cudaMemcpyAsync(&begin[0], off, 8, cudaMemcpyDefault, ctx->stream));
            CSA_CUDA(ctx, cudaMemcpyAsync(&begin[1], o, 8, cudaMemcpyDefault, ctx->stream));
            CSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            sy = sym + (begin[1] - begin[0]);
        }
        brackets_kernel<<<unsigned(div_up(c, 128)), 128, 0, ctx->stream>>>(*index, o, sy, c, brs);
        CSA_LAUNCH_CHECK(ctx);
        gather_windows_kernel<<<unsigned(div_up(c * 32, 256)), 256, 0, ctx->stream>>>(index->sa40, brs, c, win);
        CSA_LAUNCH_CHECK(ctx);
        search_windows_kernel<<<unsigned(div_up(c, 128)), 128, 0, ctx->stream>>>(*index, o, sy, c, brs, win, reinterpret_cast<u64*>(itv) + 2 * first);
        CSA_LAUNCH_CHECK(ctx);
    }
    return CSA_OK;
}

}   // namespace

extern "C" int csa_find(csa_ctx* ctx, const csa_index* index, const uint64_t* off, const uint16_t* sym, uint64_t q, uint64_t* itv)
{
    return find_batch(ctx, index, off, sym, q, itv, true);
}

extern "C" int csa_locate(csa_ctx* ctx, const csa_index* index, const uint64_t* itv, uint64_t q, uint32_t max_pos, uint64_t* pos, uint32_t* cnt)
{
    CSA_TRY(check_index(ctx, index));
    if(q == 0) return CSA_OK;
    if(!itv || !pos || !cnt || max_pos == 0) return csa_fail(ctx, CSA_E_INVALID, "csa_locate: bad argument");
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    locate_rows_kernel<<<unsigned(div_up(q * LOCATE_LANES, 256)), 256, 0, ctx->stream>>>(index->sa40, reinterpret_cast<const u64*>(itv), q, max_pos,
                                                                               reinterpret_cast<u64*>(pos), cnt);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

extern "C" int csa_certify(csa_ctx* ctx, const csa_index* index, const uint64_t* off, const uint16_t* sym, uint64_t q, const uint64_t* itv,
                           uint64_t* result)
{
    CSA_TRY(check_index(ctx, index));
    if(!result) return csa_fail(ctx, CSA_E_INVALID, "csa_certify: null result");
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    const u64 init[2] = {0, ~0ull};
    CSA_CUDA(ctx, cudaMemcpyAsync(result, init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
    CSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if(q == 0) return CSA_OK;
    if(!off || !itv) return csa_fail(ctx, CSA_E_INVALID, "csa_certify: null buffer");
    certify_kernel<<<unsigned(div_up(q, 128)), 128, 0, ctx->stream>>>(*index, reinterpret_cast<const u64*>(off), sym, q,
                                                                      reinterpret_cast<const u64*>(itv), reinterpret_cast<u64*>(result));
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

namespace
{

__global__ void add_base_kernel(u64* __restrict__ off, const u64 count, const u64 base)
{
    const u64 i = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(i < count) off[i] += base;
}

constexpr u64 HOST_CHUNK_QUERIES = u64(1) << 18;     // the reference's chunk of a host batch (include/Query_Engine.hpp:94-100)

// Device buffers of one lane of the host-batch pipeline.
struct Lane_Buffers
{
    u64* off; u16* sym; u64* itv; u32* cnt; u64* poff; u64* sums; u64* pos;
};

// ---- small host batches --------------------------------------------------------------------------------------------------------
//
// Of a batch that a warp per query answers, copies, launches and waits take longer than the search. Here it is two launches and one wait: the answers
// are written straight into pinned host memory, the positions of a query behind those of the queries before it, whose counts a block adds up by
// itself. (50 queries of up to 100 positions on 2^24 tokens: 88 us a call with five copies, six launches and two waits, this way 34 us; 1000: 92 and 43 us, 8000: 121 and 75 us.)
constexpr int ANSWER_BLOCK = 256, ANSWER_QUERIES = 32;

// What an answer goes to; cnt, pos_off and pos may be null together.
struct Answers { u64* itv; u32* cnt; u64* pos_off; u64* pos; u64 pos_capacity; u64* status; };

__global__ void __launch_bounds__(ANSWER_BLOCK) answers_kernel(const u8* __restrict__ sa40, const ulonglong2* __restrict__ itv, const u32 q, const u32 max_pos, const u64* __restrict__ status,
                                                              const Answers out)
{
    __shared__ u64 sums[ANSWER_BLOCK / 32];
    __shared__ u64 at[ANSWER_QUERIES];
    __shared__ ulonglong2 mine[ANSWER_QUERIES];
    const u32 tid = threadIdx.x, first = blockIdx.x * ANSWER_QUERIES, warp = tid >> 5;
    auto rows = [&](const ulonglong2 v) { const u64 d = v.y - v.x; return d < max_pos ? d : u64(max_pos); };
    u64 before = 0;
    if(out.pos)
    {
        for(u32 i = tid; i < first; i += ANSWER_BLOCK) before += rows(itv[i]);
        #pragma unroll
        for(int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xFFFFFFFFu, before, o);
        if(lane_id() == 0) sums[warp] = before;
        __syncthreads();
        before = 0;
        #pragma unroll
        for(int w = 0; w < ANSWER_BLOCK / 32; ++w) before += sums[w];
    }
    if(warp == 0)
    {
        const u32 i = first + tid;
        const ulonglong2 v = i < q ? itv[i] : make_ulonglong2(0, 0);
        const u64 c = out.pos ? rows(v) : 0;
        u64 inc = c;
        #pragma unroll
        for(int o = 1; o < 32; o <<= 1) { const u64 t = __shfl_up_sync(0xFFFFFFFFu, inc, o); if(int(tid) >= o) inc += t; }
        mine[tid] = v;
        at[tid] = before + inc - c;
        if(i < q)
        {
            out.itv[2 * i] = v.x;
            out.itv[2 * i + 1] = v.y;
            if(out.pos) { out.cnt[i] = u32(c); out.pos_off[i] = before + inc - c; }
            if(i == q - 1)
            {
                if(out.pos) out.pos_off[q] = before + inc;
                *out.status = *status;
            }
        }
    }
    if(!out.pos) return;
    __syncthreads();
    for(u32 k = warp; k < ANSWER_QUERIES; k += ANSWER_BLOCK / 32)
    {
        const ulonglong2 v = mine[k];
        const u64 c = rows(v), o = at[k];
        for(u64 r = lane_id(); r < c; r += 32) if(o + r < out.pos_capacity) out.pos[o + r] = sa40_load(sa40, v.x + r);
    }
}

// The address by which the device reads and writes `count` elements of host memory, null for memory that is not pinned to its end (a program may have
// registered the pages of a part of it). One question to the driver tells kind, address and range; the runtime's tells no range and takes as long.
template <typename T>
T* pinned(T* host, const u64 count)
{
    typedef CUresult (*Question)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
    static const Question ask = []() -> Question
    {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if(cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) { cudaGetLastError(); return nullptr; }
        return reinterpret_cast<Question>(f);
    }();
    if(!host || count == 0 || !ask) return nullptr;
    unsigned kind = 0, managed = 0;
    CUdeviceptr address = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute what[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED, CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                   CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* answers[5] = {&kind, &managed, &address, &start, &size};
    if(ask(5, what, answers, reinterpret_cast<CUdeviceptr>(host)) != CUDA_SUCCESS) return nullptr;
    const u64 bytes = count * sizeof(T);
    if(kind != CU_MEMORYTYPE_HOST || managed || address == 0 || address < start || address - start > size || size - (address - start) < bytes) return nullptr;
    return reinterpret_cast<T*>(address);
}

constexpr u64 STAGED_MAX = u64(1) << 20;        // bytes of a batch from or to pageable memory that are copied by way of pinned scratch
constexpr u64 READ_IN_PLACE = 256;              // queries that are read from pinned memory by the search itself: above that a copy costs less than the reads over PCIe

// A host batch of up to WARP_QUERIES queries, the array in device memory (done). Not taken: pageable buffers of a batch that is too large to be staged.
int query_host_small(csa_ctx* ctx, const csa_index* index, const u64* off_host, const u16* sym_host, const u64 q, const u32 max_pos, u64* itv_host, u32* cnt_host, u64* pos_off_host,
                     u64* pos_host, const u64 pos_capacity, u64& total, bool& done)
{
    const bool want_pos = pos_host != nullptr;
    if(off_host[q] < off_host[0]) return csa_fail(ctx, CSA_E_INVALID, "csa_query_host: offsets must not decrease");
    const u64 symbols = off_host[q] - off_host[0];
    const u64 most = want_pos ? std::min(pos_capacity, q * max_pos) : 0;
    if(symbols && !sym_host) return CSA_OK;
    u64* const pos = want_pos ? pinned(pos_host, most) : nullptr;
    if(want_pos && !pos && most * 8 > STAGED_MAX) return CSA_OK;        // before the other buffers are asked for: a question takes microseconds of a pageable one
    const u64* off = pinned(const_cast<u64*>(off_host), q + 1);
    const u16* sym = pinned(const_cast<u16*>(sym_host), symbols);
    Answers out{pinned(itv_host, 2 * q), want_pos ? pinned(cnt_host, q) : nullptr, want_pos ? pinned(pos_off_host, q + 1) : nullptr, pos, most, ctx->h_scalars + CSA_STATUS_WORD};
    // pinned scratch for what is not pinned
    const size_t b_off = off ? 0 : align_up256((q + 1) * 8), b_sym = sym || !symbols ? 0 : align_up256(symbols * 2), b_itv = out.itv ? 0 : align_up256(q * 16),
                 b_cnt = !want_pos || out.cnt ? 0 : align_up256(q * 4), b_poff = !want_pos || out.pos_off ? 0 : align_up256((q + 1) * 8),
                 b_pos = !want_pos || out.pos ? 0 : align_up256(most * 8 + 8);
    const size_t staged = b_off + b_sym + b_itv + b_cnt + b_poff + b_pos;
    if(staged > STAGED_MAX) return CSA_OK;
    void* host_ws = nullptr;
    if(staged) CSA_TRY(csa_host_aux(ctx, staged, &host_ws));
    u8* p = static_cast<u8*>(host_ws);
    if(b_off) { std::memcpy(p, off_host, (q + 1) * 8); off = reinterpret_cast<u64*>(p); p += b_off; }
    if(b_sym) { std::memcpy(p, sym_host, symbols * 2); sym = reinterpret_cast<u16*>(p); p += b_sym; }
    if(b_itv) { out.itv = reinterpret_cast<u64*>(p); p += b_itv; }
    if(b_cnt) { out.cnt = reinterpret_cast<u32*>(p); p += b_cnt; }
    if(b_poff) { out.pos_off = reinterpret_cast<u64*>(p); p += b_poff; }
    if(b_pos) out.pos = reinterpret_cast<u64*>(p);

    const size_t d_itv = align_up256(q * 16), d_off = align_up256((q + 1) * 8), d_sym = align_up256(symbols * 2 + 16);
    void* ws = nullptr;
    CSA_TRY(csa_arena(ctx, d_itv + d_off + d_sym, &ws));
    u64* const itv = static_cast<u64*>(ws);
    if(q > READ_IN_PLACE)
    {
        u64* const off_dev = reinterpret_cast<u64*>(static_cast<u8*>(ws) + d_itv);
        u16* const sym_dev = reinterpret_cast<u16*>(static_cast<u8*>(ws) + d_itv + d_off);
        CSA_CUDA(ctx, cudaMemcpyAsync(off_dev, off, (q + 1) * 8, cudaMemcpyDefault, ctx->stream));
        if(symbols) CSA_CUDA(ctx, cudaMemcpyAsync(sym_dev, sym, symbols * 2, cudaMemcpyDefault, ctx->stream));
        off = off_dev; sym = sym_dev;
    }
    find_by_warp_kernel<<<unsigned(div_up(q, 4)), 128, 0, ctx->stream>>>(*index, off, sym, q, itv);
    CSA_LAUNCH_CHECK(ctx);
    answers_kernel<<<unsigned(div_up(q, ANSWER_QUERIES)), ANSWER_BLOCK, 0, ctx->stream>>>(index->sa40, reinterpret_cast<const ulonglong2*>(itv), u32(q), max_pos, ctx->d_status, out);
    CSA_LAUNCH_CHECK(ctx);
    CSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    done = true;
    if(b_itv) std::memcpy(itv_host, out.itv, q * 16);
    if(want_pos)
    {
        total = (b_poff ? out.pos_off : pos_off_host)[q];
        if(b_cnt) std::memcpy(cnt_host, out.cnt, q * 4);
        if(b_poff) std::memcpy(pos_off_host, out.pos_off, (q + 1) * 8);
        if(b_pos && total <= most) std::memcpy(pos_host, out.pos, total * 8);
    }
    if(ctx->h_scalars[CSA_STATUS_WORD] != 0) { u64 bits = 0; return csa_sync(ctx, reinterpret_cast<uint64_t*>(&bits)); }
    return CSA_OK;
}

}   // namespace

// The host batch runs as chunks of 2^18 queries over three streams, as Query_Engine::find does (src/Query_Engine.cu:1355-1516):
// while one chunk's results cross PCIe to the host, the next chunk's search runs and the one after is on its way in. A
// chunk's positions are copied out once the host knows how many there are, one chunk behind the searches.
extern "C" int csa_query_host(csa_ctx* ctx, const csa_index* index, const uint64_t* off_host, const uint16_t* sym_host, uint64_t q, uint32_t max_pos,
                              uint64_t* itv_host, uint32_t* cnt_host, uint64_t* pos_off_host, uint64_t* pos_host, uint64_t pos_capacity,
                              uint64_t* pos_total)
{
    CSA_TRY(check_index(ctx, index));
    if(pos_total) *pos_total = 0;
    if(q == 0) return CSA_OK;
    if(!off_host || !itv_host) return csa_fail(ctx, CSA_E_INVALID, "csa_query_host: null buffer");
    const bool want_pos = max_pos > 0 && pos_host && cnt_host && pos_off_host;
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    // With the suffix array in host memory the search itself uses the context's one window buffer: one lane then.
    cudaPointerAttributes attr;
    const bool sa_on_host = cudaPointerGetAttributes(&attr, index->sa40) == cudaSuccess && attr.type == cudaMemoryTypeHost;
    cudaGetLastError();
    if(!sa_on_host && q <= WARP_QUERIES)
    {
        u64 total = 0;
        bool done = false;
        CSA_TRY(query_host_small(ctx, index, reinterpret_cast<const u64*>(off_host), sym_host, q, max_pos, reinterpret_cast<u64*>(itv_host), want_pos ? cnt_host : nullptr,
                                 want_pos ? reinterpret_cast<u64*>(pos_off_host) : nullptr, want_pos ? reinterpret_cast<u64*>(pos_host) : nullptr, pos_capacity, total, done));
        if(done)
        {
            if(pos_total && want_pos) *pos_total = total;
            if(want_pos && total > pos_capacity) return csa_fail(ctx, CSA_E_NOMEM, "csa_query_host: the positions buffer is too small");
            return CSA_OK;
        }
    }
    CSA_TRY(csa_lanes(ctx));
    const u64 chunks = div_up(q, HOST_CHUNK_QUERIES);
    const int lanes = sa_on_host ? 1 : int(chunks < u64(csa_ctx::LANES) ? chunks : u64(csa_ctx::LANES));
    const u64 cq_max = q < HOST_CHUNK_QUERIES ? q : HOST_CHUNK_QUERIES;
    u64 sym_max = 0;
    for(u64 c = 0; c < chunks; ++c)
    {
        const u64 first = c * HOST_CHUNK_QUERIES, cq = (q - first < HOST_CHUNK_QUERIES ? q - first : HOST_CHUNK_QUERIES);
        if(off_host[first + cq] < off_host[first]) return csa_fail(ctx, CSA_E_INVALID, "csa_query_host: offsets must not decrease");
        const u64 sc = off_host[first + cq] - off_host[first];
        if(sc > sym_max) sym_max = sc;
    }
    const size_t b_off = align_up256((cq_max + 1) * 8), b_sym = align_up256(sym_max * 2 + 16), b_itv = align_up256(cq_max * 16), b_cnt = align_up256(cq_max * 4),
                 b_poff = align_up256((cq_max + 1) * 8), b_sums = align_up256((div_up(cq_max, SCAN_TILE) + 1) * 8),
                 b_pos = want_pos ? align_up256(size_t(cq_max) * max_pos * 8) : 0;
    const size_t per_lane = b_off + b_sym + b_itv + b_cnt + b_poff + b_sums + b_pos;
    void* ws = nullptr;
    CSA_TRY(csa_arena(ctx, per_lane * lanes + 4096, &ws));
    Lane_Buffers L[csa_ctx::LANES];
    for(int l = 0; l < lanes; ++l)
    {
        u8* p = static_cast<u8*>(ws) + per_lane * l;
        L[l].off = reinterpret_cast<u64*>(p); p += b_off;
        L[l].sym = reinterpret_cast<u16*>(p); p += b_sym;
        L[l].itv = reinterpret_cast<u64*>(p); p += b_itv;
        L[l].cnt = reinterpret_cast<u32*>(p); p += b_cnt;
        L[l].poff = reinterpret_cast<u64*>(p); p += b_poff;
        L[l].sums = reinterpret_cast<u64*>(p); p += b_sums;
        L[l].pos = reinterpret_cast<u64*>(p);
    }
    CSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));       // whatever the caller queued on the context's own stream comes first

    // search of chunk c: batch in, intervals out, counts, offsets inside the chunk, positions packed in the lane's buffer
    auto search = [&](u64 c) -> int
    {
        const int l = int(c % u64(lanes));
        const u64 first = c * HOST_CHUNK_QUERIES, cq = (q - first < HOST_CHUNK_QUERIES ? q - first : HOST_CHUNK_QUERIES);
        const u64 sc = off_host[first + cq] - off_host[first];
        const On_Stream on(ctx, ctx->lane[l]);
        CSA_CUDA(ctx, cudaMemcpyAsync(L[l].off, off_host + first, (cq + 1) * 8, cudaMemcpyHostToDevice, ctx->stream));
        if(sc) CSA_CUDA(ctx, cudaMemcpyAsync(L[l].sym, sym_host + (off_host[first] - off_host[0]), sc * 2, cudaMemcpyHostToDevice, ctx->stream));
        CSA_TRY(find_batch(ctx, index, reinterpret_cast<uint64_t*>(L[l].off), L[l].sym, cq, reinterpret_cast<uint64_t*>(L[l].itv), false));
        CSA_CUDA(ctx, cudaMemcpyAsync(itv_host + 2 * first, L[l].itv, cq * 16, cudaMemcpyDeviceToHost, ctx->stream));
        if(want_pos)
        {
            counts_kernel<<<unsigned(div_up(cq, 256)), 256, 0, ctx->stream>>>(L[l].itv, cq, max_pos, L[l].cnt);
            CSA_LAUNCH_CHECK(ctx);
            u64* total_d = ctx->d_scalars + 8 + l;
            CSA_TRY(exclusive_sum(ctx, L[l].cnt, cq, L[l].poff, L[l].sums, total_d));
            locate_packed_kernel<<<unsigned(div_up(cq * LOCATE_LANES, 256)), 256, 0, ctx->stream>>>(index->sa40, L[l].itv, cq, max_pos, L[l].poff, L[l].pos);
            CSA_LAUNCH_CHECK(ctx);
            CSA_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + 8 + l, total_d, 8, cudaMemcpyDeviceToHost, ctx->stream));
            CSA_CUDA(ctx, cudaMemcpyAsync(cnt_host + first, L[l].cnt, cq * 4, cudaMemcpyDeviceToHost, ctx->stream));
        }
        CSA_CUDA(ctx, cudaEventRecord(ctx->lane_event[l], ctx->stream));
        return CSA_OK;
    };
    // delivery of chunk c, once its search is over: its positions go behind those of the chunks before it
    u64 base = 0;
    bool overflow = false;
    auto deliver = [&](u64 c) -> int
    {
        if(!want_pos) return CSA_OK;
        const int l = int(c % u64(lanes));
        const u64 first = c * HOST_CHUNK_QUERIES, cq = (q - first < HOST_CHUNK_QUERIES ? q - first : HOST_CHUNK_QUERIES);
        CSA_CUDA(ctx, cudaEventSynchronize(ctx->lane_event[l]));
        const u64 total = ctx->h_scalars[8 + l];
        const On_Stream on(ctx, ctx->lane[l]);
        if(base)
        {
            add_base_kernel<<<unsigned(div_up(cq, 256)), 256, 0, ctx->stream>>>(L[l].poff, cq, base);
            CSA_LAUNCH_CHECK(ctx);
        }
        CSA_CUDA(ctx, cudaMemcpyAsync(pos_off_host + first, L[l].poff, cq * 8, cudaMemcpyDeviceToHost, ctx->stream));
        if(base + total > pos_capacity) overflow = true;
        else if(total) CSA_CUDA(ctx, cudaMemcpyAsync(pos_host + base, L[l].pos, total * 8, cudaMemcpyDeviceToHost, ctx->stream));
        base += total;
        return CSA_OK;
    };
    // With two or more lanes the delivery of a chunk is issued after the search of the next one (which runs on another lane);
    // one lane takes the chunks one by one.
    const bool pipelined = lanes >= 2;
    int rc = CSA_OK;
    for(u64 c = 0; c < chunks && rc == CSA_OK; ++c)
    {
        rc = search(c);
        if(rc != CSA_OK) break;
        if(!pipelined) rc = deliver(c);
        else if(c >= 1) rc = deliver(c - 1);
    }
    if(rc == CSA_OK && pipelined) rc = deliver(chunks - 1);
    for(int l = 0; l < lanes; ++l) cudaStreamSynchronize(ctx->lane[l]);      // on every path: the lanes' buffers are the arena's
    CSA_TRY(rc);
    if(want_pos)
    {
        pos_off_host[q] = base;
        if(pos_total) *pos_total = base;
        if(overflow) return csa_fail(ctx, CSA_E_NOMEM, "csa_query_host: the positions buffer is too small");
    }
    u64 bits = 0;
    return csa_sync(ctx, reinterpret_cast<uint64_t*>(&bits));
}
