// What follows generation 0 of the resident build: tied suffixes are ordered group by group. A group of up to SMALL_GROUP
// suffixes never meets a radix sort: its records lie side by side in a list, a block takes a window of the list into shared
// memory, and every record counts the smaller members of its own group. That costs one read and one write of the list plus the
// random read of what the records are compared by, where a radix sort of the whole list moves every record eight times.
//
// Compared are first the symbols themselves (a few 16-byte words of text per suffix settle all ties of a text without long
// repeats; no inverse array is made at all then), later, where long repeats leave ties, the ranks of the suffixes h symbols
// further on (prefix doubling, as the reference's generations t >= 1, src/GPU_SACA.cu:1714-1995).
#include "part.cuh"
#include "refine.cuh"

namespace
{

constexpr int RW_BLOCK = 256, RW_ITEMS = 8, RW_WINDOW = RW_BLOCK * RW_ITEMS;
constexpr u32 RW_TILE = RW_WINDOW - SMALL_GROUP;        // groups that start in the tile end inside the window
constexpr u32 NO_GROUP = 0xFFFFu;

__device__ __forceinline__ u32 warp_sum(u32 v)
{
    #pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const u32 t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if(int(lane_id()) >= o) v += t;
    }
    return v;
}

// Groups of a block's window of a list (slot j = entry first + j), found by bit operations: bit j of `starts` says that a group (or
// what lies past the list's end) begins at slot j.
struct Group_Starts
{
    u32 starts[RW_WINDOW / 32];
};

// A thread's records are the slots tid + i * RW_BLOCK: e[i] gets the entries (~0 past the list's end: no group starts at slot
// 2^32 - 1). Ends with a barrier.
__device__ __forceinline__ void load_entries(Group_Starts& g, const u64* __restrict__ list, const u64 count, const u64 first, u64 (&e)[RW_ITEMS])
{
    const u32 tid = threadIdx.x, lane = lane_id();
    u32 before[RW_ITEMS];       // of lane 0: the head before its slot
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u64 k = first + tid + i * RW_BLOCK;
        e[i] = k < count ? list[k] : ~0ull;
        before[i] = 0xFFFFFFFEu;        // another number than any head
        if(lane == 0 && k > 0) before[i] = k - 1 < count ? u32(list[k - 1] >> 32) : 0xFFFFFFFFu;
    }
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 h = u32(e[i] >> 32), up = __shfl_up_sync(0xFFFFFFFFu, h, 1);
        const u32 m = __ballot_sync(0xFFFFFFFFu, h != (lane ? up : before[i]));
        if(lane == 0) g.starts[i * (RW_BLOCK / 32) + (tid >> 5)] = m;
    }
    __syncthreads();
}

// First and end slot of the group of slot tid + i * RW_BLOCK; first = NO_GROUP where the group does not start inside the block's
// tile (it belongs to another block) or the slot lies past the list's end. Every lane of a warp calls it.
__device__ __forceinline__ void find_group(const Group_Starts& g, const u64 entry, const int i, u32& s, u32& e)
{
    const u32 lane = lane_id();
    const int word = i * (RW_BLOCK / 32) + int(threadIdx.x >> 5);
    s = NO_GROUP; e = 0;
    if(__all_sync(0xFFFFFFFFu, entry == ~0ull)) return;
    const u32 m = g.starts[word];
    u32 last = NO_GROUP, next = RW_WINDOW;      // of the words before and behind: the same for all lanes
    constexpr int REACH = SMALL_GROUP / 32 + 1;
    if((m & 1u) == 0)
        for(int k = word - 1; k >= 0 && k >= word - REACH; --k)
            if(const u32 v = g.starts[k]) { last = k * 32 + 31 - __clz(v); break; }
    for(int k = word + 1; k < RW_WINDOW / 32 && k <= word + REACH; ++k)
        if(const u32 v = g.starts[k]) { next = k * 32 + __ffs(v) - 1; break; }
    const u32 upto = m & (0xFFFFFFFFu >> (31 - lane)), behind = m & ~(0xFFFFFFFFu >> (31 - lane));
    s = upto ? word * 32 + 31 - __clz(upto) : last;
    e = behind ? word * 32 + __ffs(behind) - 1 : next;
    if(s >= RW_TILE || entry == ~0ull) s = NO_GROUP;
}

// Where the members of a window's groups go, found without comparing all with all: most members of a group equal its first member
// (in near-duplicate documents two copies differ in one symbol of a thousand), and only the others, the odd ones, are counted
// against one another.
struct Odd_Members
{
    u32 odd[RW_WINDOW / 32 + 1];            // a bit per slot: another key than the group's first member
    u32 less[RW_WINDOW / 32 + 1];           // of those, the smaller ones
    u32 before[RW_WINDOW / 32 + 1];         // per word: odd members before it | smaller ones before it << 16
};

// The bits of slot tid + i * RW_BLOCK; every lane calls it.
__device__ __forceinline__ void mark_odd(Odd_Members& m, const int i, const bool odd, const bool less)
{
    const u32 o = __ballot_sync(0xFFFFFFFFu, odd), l = __ballot_sync(0xFFFFFFFFu, less);
    if(lane_id() == 0) { m.odd[i * (RW_BLOCK / 32) + (threadIdx.x >> 5)] = o; m.less[i * (RW_BLOCK / 32) + (threadIdx.x >> 5)] = l; }
}

// Between barriers: the sums over the words.
__device__ __forceinline__ void sum_odd(Odd_Members& m)
{
    static_assert(RW_WINDOW / 32 == 64, "two words a lane");
    if(threadIdx.x < 32)
    {
        const u32 k = 2 * threadIdx.x;
        const u32 a = __popc(m.odd[k]) | __popc(m.less[k]) << 16, b = __popc(m.odd[k + 1]) | __popc(m.less[k + 1]) << 16;
        const u32 inc = warp_sum(a + b);
        m.before[k] = inc - a - b;
        m.before[k + 1] = inc - b;
        if(threadIdx.x == 31) { m.before[64] = inc; m.odd[64] = 0; m.less[64] = 0; }
    }
}

// Odd members before slot j | smaller ones << 16 (j up to RW_WINDOW).
__device__ __forceinline__ u32 odd_before(const Odd_Members& m, const u32 j)
{
    const u32 below = (1u << (j & 31)) - 1;
    return m.before[j >> 5] + (__popc(m.odd[j >> 5] & below) | __popc(m.less[j >> 5] & below) << 16);
}

// How many of the odd keys [a, b) are smaller than `mine`, how many equal it, and how many of those come before entry `me`: in bits
// 0, 16 and 32 on. A call, so that the eight places that need it do not each carry the loop (instruction fetch bounds the callers).
template <typename K>
__device__ __noinline__ u64 count_odd(const K* keys, const u32 a, const u32 b, const u32 me, const K mine)
{
    u32 less = 0, eq_before = 0, eq = 0;
    for(u32 k = a; k < b; ++k)
    {
        const K o = keys[k];
        less += o < mine;
        const u32 same = o == mine;
        eq += same;
        eq_before += same && k < me;
    }
    return u64(less | eq << 16) | u64(eq_before) << 32;
}

// The place of member j of the group [s, e), and the new group that it lands in. keys: the odd members' keys, side by side in slot order.
template <typename K>
__device__ __forceinline__ void member_place(const Odd_Members& m, const K* keys, const u32 j, const u32 s, const u32 e, const bool odd, const bool smaller, const K mine,
                                             u32& at, u32& to_s, u32& to_e)
{
    const u32 bs = odd_before(m, s), be = odd_before(m, e), bj = odd_before(m, j);
    const u32 equals = (e - s) - ((be - bs) & 0xFFFFu);
    if(!odd)
    {
        to_s = s + ((be >> 16) - (bs >> 16));
        to_e = to_s + equals;
        at = to_s + (j - s) - ((bj - bs) & 0xFFFFu);
        return;
    }
    const u64 c = count_odd(keys, bs & 0xFFFFu, be & 0xFFFFu, bj & 0xFFFFu, mine);
    const u32 less = u32(c) & 0xFFFFu, eq = u32(c) >> 16, eq_before = u32(c >> 32);
    to_s = s + less + (smaller ? 0 : equals);
    at = to_s + eq_before;
    to_e = to_s + eq;
}

// The window of a list with its groups in shared memory, where a kernel changes them: gs[j]: first slot of j's group or NO_GROUP;
// ge[gs[j]]: where the group ends; head[j]: j's place in the suffix array.
struct Window
{
    Group_Starts groups;
    u32 head[RW_WINDOW];
    u32 pos[RW_WINDOW];
    u16 gs[RW_WINDOW];
    u16 ge[RW_WINDOW];
    u32 mask[RW_WINDOW / 32];
    u32 pre[RW_WINDOW / 32];
    u32 warp_tot[RW_BLOCK / 32];
    u32 slot;
};

// Ends with a barrier.
__device__ __forceinline__ void load_window(Window& w, const u64* __restrict__ list, const u64 count, const u64 first)
{
    u64 entry[RW_ITEMS];
    load_entries(w.groups, list, count, first, entry);
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = threadIdx.x + i * RW_BLOCK;
        u32 s, e;
        find_group(w.groups, entry[i], i, s, e);
        w.head[j] = u32(entry[i] >> 32) + (s == NO_GROUP ? 0 : j - s);
        w.pos[j] = u32(entry[i]);
        w.gs[j] = u16(s);
        if(s == j) w.ge[j] = u16(e);
    }
    __syncthreads();
}

// Appends the slots flagged in w.mask (cleared before, set by atomics, no barrier needed in between) to a list whose length
// *count is advanced; returns the list position of the first. Every thread calls it; the result holds after the call. W: a struct
// with mask, pre, warp_tot and slot as in Window.
template <typename W>
__device__ __forceinline__ u32 window_places(W& w, u32* count)
{
    __syncthreads();
    constexpr int WORDS = RW_WINDOW / 32;       // 64
    const u32 tid = threadIdx.x;
    const u32 c = tid < WORDS ? __popc(w.mask[tid]) : 0;
    const u32 inc = warp_sum(c);
    if(lane_id() == 31) w.warp_tot[tid >> 5] = inc;
    __syncthreads();
    if(tid < WORDS) w.pre[tid] = inc - c + (tid >= 32 ? w.warp_tot[0] : 0);
    if(tid == 0) { const u32 total = w.warp_tot[0] + w.warp_tot[1]; w.slot = total ? atomicAdd(count, total) : 0; }
    __syncthreads();
    return w.slot;
}

__device__ __forceinline__ u32 swap_halves(u32 x) { return __funnelshift_l(x, x, 16); }

// Eight symbols from text position x on, most significant first; symbols past the text's end are 0 (x < n: the text is padded).
__device__ __forceinline__ ulonglong2 eight_symbols(const u16* __restrict__ T, const u64 x)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(T + x);
    const uint2* p = reinterpret_cast<const uint2*>(a & ~uintptr_t(7));
    const uint2 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2);
    const u32 sh = u32(a & 3) * 8;                // 0 or 16
    const u32 w[6] = {q0.x, q0.y, q1.x, q1.y, q2.x, q2.y};
    const bool odd = (a & 4) != 0;
    u32 v[5], r[4];
    #pragma unroll
    for(int k = 0; k < 5; ++k) v[k] = odd ? w[k + 1] : w[k];
    #pragma unroll
    for(int k = 0; k < 4; ++k) r[k] = swap_halves(__funnelshift_r(v[k], v[k + 1], sh));
    return make_ulonglong2((u64(r[0]) << 32) | r[1], (u64(r[2]) << 32) | r[3]);
}

// How a member of a group compares with the group's first member from the group's depth on, as one number that orders the members:
// class (0 less, 1 equal as far as compared, 2 greater) at bit 40, then the pair of symbols in which the two differ first (more
// equal pairs: nearer to the first member), then that pair and how many symbols of it the suffix has.
constexpr u64 KEY_EQUAL = 1ull << 40;

__device__ __forceinline__ u64 pair_key(const u32 pair, const u32 mine, const u32 have, const u32 lead, const u32 lead_have)
{
    const bool less = mine < lead || (mine == lead && have < lead_have);
    return (less ? 0ull : 2ull << 40) | (u64(less ? pair : 31 - pair) << 34) | (u64(mine) << 2) | have;
}
// Symbols that members with this key share beyond the group's depth (`reach`: as far as was compared).
__device__ __forceinline__ u32 shared_by_key(const u64 key, const u32 reach)
{
    if(key == KEY_EQUAL) return reach;
    const u32 p = u32(key >> 34) & 31u;
    return 2 * ((key >> 40) ? 31 - p : p) + 2;
}

constexpr u32 WIDE_REACH = 48;      // symbols that four lanes compare at once: 64, of which up to 15 lie before the suffix
constexpr u32 QUICK_REACH = 8;
constexpr int WIDE_ROWS = 2;         // suffixes in flight per four lanes
static_assert(TEXT_DEPTH == 1 + WIDE_REACH, "one wide round");

// 32 bytes, a whole sector, by one load.
struct Piece { u32 w[8]; };
__device__ __forceinline__ Piece load_sector(const uintptr_t at)
{
    Piece p;
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(p.w[0]), "=r"(p.w[1]), "=r"(p.w[2]), "=r"(p.w[3]), "=r"(p.w[4]), "=r"(p.w[5]), "=r"(p.w[6]), "=r"(p.w[7]) : "l"(at));
    return p;
}

// Where the suffixes at x and y first differ, among 16 of their symbols: those of the part-th sector that holds symbols of the suffix at x. `none` where they
// do not below symbol `limit`. The other suffix comes in pieces of 16 bytes that are shifted to meet the sector. The first sector may begin up to
// 15 symbols before x, inside the allocation, as it holds x; pieces of 16 bytes before the text are not read; behind it the text is padded.
__device__ __forceinline__ u32 first_difference(const u16* __restrict__ T, const u64 x, const u64 y, const u32 part, const u32 limit, const u32 none)
{
    const uintptr_t at = reinterpret_cast<uintptr_t>(T + x), text = reinterpret_cast<uintptr_t>(T);
    const u32 skip = u32(at >> 1) & 15u;
    const int base = int(16 * part) - int(skip);
    if(base >= int(limit)) return none;
    const Piece a = load_sector((at & ~uintptr_t(31)) + 32 * part);
    const uintptr_t from = reinterpret_cast<uintptr_t>(T + y) - 2 * skip + 32 * part, piece = from & ~uintptr_t(15);
    const u32 shift = u32(from >> 1) & 7u;
    auto load = [&](const uintptr_t q) { return q >= text ? __ldg(reinterpret_cast<const uint4*>(q)) : make_uint4(0, 0, 0, 0); };      // T is 16-byte aligned
    const uint4 w0 = load(piece), w1 = load(piece + 16), w2 = load(piece + 32);
    u32 v[12] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x, w2.y, w2.z, w2.w};
    #pragma unroll
    for(int k = 0; k < 10; ++k) v[k] = (shift & 4) ? v[k + 2] : v[k];
    #pragma unroll
    for(int k = 0; k < 9; ++k) v[k] = (shift & 2) ? v[k + 1] : v[k];
    u32 any = 0;
    #pragma unroll
    for(int k = 0; k < 8; ++k) { v[k] = __funnelshift_r(v[k], v[k + 1], (shift & 1) * 16) ^ a.w[k]; any |= v[k]; }
    if(any == 0) return none;
    u32 differ = 0;
    #pragma unroll
    for(int k = 0; k < 8; ++k) differ |= ((v[k] & 0xFFFFu) ? 1u << (2 * k) : 0u) | ((v[k] >> 16) ? 2u << (2 * k) : 0u);
    if(base < 0) differ &= ~0u << -base;
    const u32 first = u32(base + __ffs(differ) - 1);
    return differ && first < limit ? first : none;
}

// The key of the suffix at x, of which cx symbols count, against the one at y, with cy: they differ first at symbol `first`, or one ends there.
__device__ __forceinline__ u64 difference_key(const u16* __restrict__ T, const u64 x, const u64 y, const u32 cx, const u32 cy, const u32 first)
{
    const u32 pair = first >> 1;
    auto two = [&](const u64 z, const u32 c, u32& have) -> u32         // the pair of symbols, most significant first
    {
        const u32 at = 2 * pair;
        have = c > at + 1 ? 2 : (c > at ? 1 : 0);
        return (have ? u32(T[z + at]) << 16 : 0u) | (have > 1 ? u32(T[z + at + 1]) : 0u);
    };
    u32 hx, hy;
    const u32 mine = two(x, cx, hx), lead = two(y, cy, hy);
    return pair_key(pair, mine, hx, lead, hy);
}

// A sample of a list of small groups, a warp to an entry: whether all suffixes of the entry's group still have one key one symbol on, by their symbols' code words (a key is
// key_bits bits), and whether the entry beside it shares `depth` symbols with it. A function of its own: it takes no registers from the kernel that calls it.
__device__ __noinline__ void sample_ties(const u64* __restrict__ list, const u64 count, const u16* __restrict__ T, const u64 n, const u32* __restrict__ code, const u32 key_bits, const u32 depth,
                                         Build_Counts* __restrict__ counts)
{
    const u64 step = (count + TIE_SAMPLE - 1) / TIE_SAMPLE;
    auto symbol = [&](const u64 at) { return at < n ? u32(__ldg(T + at)) : 0u; };
    for(u64 k = (u64(blockIdx.x) * (RW_BLOCK / 32) + (threadIdx.x >> 5)) * step; k < count; k += u64(gridDim.x) * (RW_BLOCK / 32) * step)
    {
        const u64 e = __ldg(list + k), x = u32(e);
        constexpr int PIECES = 2 * int(SMALL_GROUP) / 32;       // the entries before and behind: a small group reaches no further
        u64 near[PIECES];
        #pragma unroll
        for(int c = 0; c < PIECES; ++c)
        {
            const long long at = (long long)(k) - int(SMALL_GROUP) + c * 32 + int(lane_id());
            near[c] = at >= 0 && u64(at) < count && u64(at) != k ? __ldg(list + at) : ~e;
        }
        // The group's keys tell its first `whole` symbols, the keys one symbol on end before symbol `end`. A lane reads two code words, of a bit or more: a key has no more of them.
        const u32 w0 = __ldg(code + symbol(x + lane_id())) & 31u, w1 = __ldg(code + symbol(x + 32 + lane_id())) & 31u;
        const u32 to0 = warp_sum(w0), to1 = warp_sum(w1) + __shfl_sync(0xFFFFFFFFu, to0, 31), first = __shfl_sync(0xFFFFFFFFu, w0, 0);
        auto symbols_upto = [&](const u32 bits) { return u32(__popc(__ballot_sync(0xFFFFFFFFu, to0 <= bits)) + __popc(__ballot_sync(0xFFFFFFFFu, to1 <= bits))); };
        const u32 whole = max(1u, symbols_upto(key_bits)), end = symbols_upto(key_bits + first - 1) + 1;
        const u32 last = whole - 1, upto0 = __shfl_sync(0xFFFFFFFFu, to0, last & 31), upto1 = __shfl_sync(0xFFFFFFFFu, to1, last & 31);
        const u32 before = (last < 32 ? upto0 : upto1) - first;         // bits from symbol 1 up to symbol `whole`
        bool leaves = false, any = false;
        #pragma unroll
        for(int c = 0; c < PIECES; ++c)
        {
            if(u32(near[c] >> 32) != u32(e >> 32)) continue;
            any = true;
            const u64 y = u32(near[c]);
            u32 upto = before;
            for(u32 d = whole; d < end; ++d)
            {
                const u32 a = __ldg(code + symbol(x + d)), b = __ldg(code + symbol(y + d));
                if(a != b) { leaves |= upto + __clz((a ^ b) & ~31u) < key_bits; break; }
                upto += a & 31u;
            }
        }
        leaves = __any_sync(0xFFFFFFFFu, leaves);
        any = __any_sync(0xFFFFFFFFu, any);
        const u64 behind = __shfl_sync(0xFFFFFFFFu, near[PIECES / 2], 1), ahead = __shfl_sync(0xFFFFFFFFu, near[PIECES / 2 - 1], 31);
        const u64 y = u32(u32(behind >> 32) == u32(e >> 32) ? behind : ahead);
        bool differs = false;
        for(u32 d = lane_id(); d < depth; d += 32) differs |= x + d >= n || y + d >= n || T[x + d] != T[y + d];
        differs = __any_sync(0xFFFFFFFFu, differs);
        if(lane_id() == 0 && any)
        {
            atomicAdd(&counts->looked_at, 1u);
            if(!leaves) atomicAdd(&counts->lead_on, 1u);
            if(!differs) atomicAdd(&counts->far_ties, 1u);
        }
    }
}

// A list of few entries whose groups have up to NARROW_GROUP members, in the first round, up to symbol TEXT_DEPTH: a thread for an entry compares its suffix with the others of its group, eight symbols at a
// time. What the kernel below takes is mostly the fetching of its instructions and a chain of steps then: 2^18 tokens 14.7 us, this way 6.5; 2^24 24 and 8.5 (a build 459 and 441). What is left to the
// rounds behind that is alike for hundreds of symbols, and a thread would read all of them, of every other member, one after the other: 1e7 tokens with a passage of 1500 fifteen times 6.29 ms a build,
// with one of 500 1.79; by the kernel below from the second round on 1.23 and 0.74. Two copies of 500 take 0.49 and 0.54.
constexpr u32 NARROW_MOST = 1u << 15;

// -1, 0, 1: the suffix at x comes before the one at y, shares symbols [from, to) with it, comes behind it.
__device__ __forceinline__ int compare_suffixes(const u16* __restrict__ T, const u64 n, u64 x, u64 y, const u64 from, const u64 to)
{
    x += from; y += from;
    for(u64 d = from; d < to; d += 8, x += 8, y += 8)
    {
        const u32 most = u32(min(to - d, u64(8))), has_x = x < n ? u32(min(n - x, u64(most))) : 0u, has_y = y < n ? u32(min(n - y, u64(most))) : 0u, both = min(has_x, has_y);
        if(both)
        {
            const ulonglong2 a = eight_symbols(T, x), b = eight_symbols(T, y);
            const u64 high = a.x ^ b.x, low = a.y ^ b.y;
            const u32 first = high ? __clzll(high) / 16 : 4 + (low ? __clzll(low) / 16 : 4);
            if(first < both) return (high ? a.x < b.x : a.y < b.y) ? -1 : 1;
        }
        if(has_x != has_y) return has_x < has_y ? -1 : 1;
    }
    return 0;
}

__device__ __noinline__ void refine_narrow(const u16* __restrict__ T, const u64 n, const u64 from, const u64 to, const u64* __restrict__ list, const u32 count, u64* __restrict__ next, u32* __restrict__ sa,
                                           u8* __restrict__ sa40, Build_Counts* __restrict__ counts)
{
    for(u32 i = blockIdx.x * RW_BLOCK + threadIdx.x; i < count; i += gridDim.x * RW_BLOCK)
    {
        const u64 mine = list[i];
        const u32 head = u32(mine >> 32), x = u32(mine);
        u32 first = i;
        while(first > 0 && i - first < NARROW_GROUP && u32(list[first - 1] >> 32) == head) --first;
        u32 less = 0, same = 0;         // members that come before; a bit for each that is still tied with this one
        for(u32 j = first; j < count && j - first < NARROW_GROUP; ++j)
        {
            const u64 other = list[j];
            if(u32(other >> 32) != head) break;
            if(j == i) continue;
            const int c = compare_suffixes(T, n, x, u32(other), from, to);
            less += c > 0;
            same |= u32(c == 0) << (j - first);
        }
        const u32 place = head + less;
        if(same == 0)
        {
            if(sa) sa[place] = x;
            else
            {
                u8* const at = sa40 + 5 * u64(place);
                at[0] = u8(x); at[1] = u8(x >> 8); at[2] = u8(x >> 16); at[3] = u8(x >> 24); at[4] = 0;
            }
        }
        else if((same & ((1u << (i - first)) - 1)) == 0)        // the first of a group writes it
        {
            u32 at = atomicAdd(&counts->next_small, u32(__popc(same)) + 1);
            next[at++] = u64(place) << 32 | x;
            for(; same; same &= same - 1) next[at++] = u64(place) << 32 | u32(list[first + __ffs(same) - 1]);
        }
    }
}

// Orders groups by the symbols [from, to) of their suffixes. In a round every member of a group is compared with the group's first
// member, and the members are put in order by their first difference from it; a group that falls apart goes on as several, each
// with its own depth. The window stays in shared memory over all rounds.
//
// A WIDE round compares 48 symbols: four lanes read a suffix, a sector each, all of it in flight at once, and the first member's symbols beside it, which the
// neighbouring lanes read as well; a difference is then read symbol by symbol. (Half a warp to a suffix, four symbols a lane: 58 warp instructions a suffix,
// 9.45 ms for 10^8 near-duplicate suffixes; a thread to a suffix, a sector after the other: 11.5 ms; this way 8.9 ms, and 7.8 ms
// with what is done with passed over.)
// Where few suffixes are tied, nearly all of them differ within a few symbols and
// the chain of loads counts: the first round is then QUICK, 8 symbols by one thread, all of a thread's suffixes in flight together.
__global__ void __launch_bounds__(RW_BLOCK, 4) refine_by_text_kernel(const u16* __restrict__ T, const u64 n, const u64 from, const u64 to, const u64* __restrict__ list,
                                                                    u64* __restrict__ next, u32* __restrict__ sa, u8* __restrict__ sa40, u32* __restrict__ isa, Build_Counts* __restrict__ counts,
                                                                    const u64 most, const u32* __restrict__ code, const u32 key_bits)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Window& w = *reinterpret_cast<Window*>(smem_raw);
    u64* const key = reinterpret_cast<u64*>(smem_raw + (sizeof(Window) + 15) / 16 * 16);     // [RW_WINDOW]
    u32* const depth = reinterpret_cast<u32*>(key + RW_WINDOW);     // [RW_WINDOW] by first slot: symbols that the group's members share (below 2^32: no more than n)
    Odd_Members& odds = *reinterpret_cast<Odd_Members*>(depth + RW_WINDOW);
    const u32 tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    wait_for_previous();
    if(counts->oversize != 0) return;           // children still wait for the radix sort: their records lie where `next` would go
    const u64 count = counts->small;
    if(to <= TEXT_DEPTH && count <= NARROW_MOST && counts->wide == 0 && isa == nullptr && count <= most)
    {
        refine_narrow(T, n, from, to, list, u32(count), next, sa, sa40, counts);
        return;
    }
    if(count > most)
    {
        if(code != nullptr) sample_ties(list, count, T, n, code, key_bits, u32(to), counts);
        return;
    }
    for(u64 first = u64(blockIdx.x) * RW_TILE; first < count; first += u64(gridDim.x) * RW_TILE)
    {
        load_window(w, list, count, first);
        #pragma unroll
        for(int i = 0; i < RW_ITEMS; ++i) depth[tid + i * RW_BLOCK] = u32(from);
        __syncthreads();
        int quick = from < QUICK_REACH && to - from >= 2 * QUICK_REACH && count * 4 < n ? 2 : 0;       // rounds of that kind
        bool again = false;
        while(true)
        {
            const u32 reach = quick ? QUICK_REACH : WIDE_REACH;
            // w.mask: the slots of groups that go on. Most groups are done with after the first round, and a warp passes over words without such a slot.
            u32 open = 0;           // the thread's, a bit per item
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
            {
                const u32 word = i * (RW_BLOCK / 32) + warp;
                if(again && w.mask[word] == 0) continue;
                const u32 s = w.gs[tid + i * RW_BLOCK];
                const bool mine = s != NO_GROUP && u32(w.ge[s]) - s >= 2 && u64(depth[s]) < to;
                const u32 all = __ballot_sync(0xFFFFFFFFu, mine);
                if(lane == 0) w.mask[word] = all;
                open |= u32(mine) << i;
            }
            again = true;
            if(!__syncthreads_or(open != 0)) break;
            if(quick)
            {
                #pragma unroll 4
                for(int i = 0; i < RW_ITEMS; ++i)
                {
                    const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
                    if((open >> i & 1u) == 0) continue;
                    if(j == s) { key[j] = KEY_EQUAL; continue; }
                    const u64 x = u64(w.pos[j]) + depth[s], y = u64(w.pos[s]) + depth[s];
                    const ulonglong2 none = make_ulonglong2(0, 0);
                    const ulonglong2 a = x < n ? eight_symbols(T, x) : none, b = y < n ? eight_symbols(T, y) : none;
                    const u64 has_a = x < n ? n - x : 0, has_b = y < n ? n - y : 0;
                    const u32 pa[4] = {u32(a.x >> 32), u32(a.x), u32(a.y >> 32), u32(a.y)}, pb[4] = {u32(b.x >> 32), u32(b.x), u32(b.y >> 32), u32(b.y)};
                    u64 k = KEY_EQUAL;
                    #pragma unroll
                    for(int q = 3; q >= 0; --q)
                    {
                        const u32 ha = has_a > 2 * q + 1 ? 2 : (has_a > 2 * q ? 1 : 0), hb = has_b > 2 * q + 1 ? 2 : (has_b > 2 * q ? 1 : 0);
                        if(pa[q] != pb[q] || ha != hb) k = pair_key(q, pa[q], ha, pb[q], hb);
                    }
                    key[j] = k;
                }
            }
            else
            {
                const u32 part = lane & 3u, quad = lane & ~3u;
                #pragma unroll (WIDE_ROWS)
                for(u32 j0 = warp * 8; j0 < RW_WINDOW; j0 += RW_BLOCK / 4)
                {
                    const u32 eight = w.mask[j0 >> 5] >> (j0 & 31) & 0xFFu, j = j0 + (lane >> 2);
                    if(eight == 0) continue;
                    bool mine = eight >> (lane >> 2) & 1u;
                    const u32 s = mine ? u32(w.gs[j]) : 0u;
                    if(mine && j == s && part == 0) key[j] = KEY_EQUAL;
                    mine = mine && j != s;
                    const u64 d = depth[s];
                    u64 x = 0, y = 0;
                    u32 cx = 0, cy = 0, first = WIDE_REACH;
                    if(mine)
                    {
                        x = w.pos[j] + d; y = w.pos[s] + d;
                        const u64 most = min(to - d, u64(WIDE_REACH));
                        cx = x < n ? u32(min(n - x, most)) : 0u;
                        cy = y < n ? u32(min(n - y, most)) : 0u;
                        first = first_difference(T, x, y, part, min(cx, cy), WIDE_REACH);
                    }
                    const u32 found = __ballot_sync(0xFFFFFFFFu, first != WIDE_REACH) >> quad & 15u;
                    if(mine && part == (found ? u32(__ffs(found)) - 1 : 0u))
                        key[j] = found || cx != cy ? difference_key(T, x, y, cx, cy, found ? first : min(cx, cy)) : KEY_EQUAL;
                }
            }
            __syncthreads();
            // the members take their new places
            u64 mine[RW_ITEMS];
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
            {
                const u32 word = i * (RW_BLOCK / 32) + warp;
                mine[i] = KEY_EQUAL;
                if(w.mask[word] == 0)
                {
                    if(lane == 0) { odds.odd[word] = 0; odds.less[word] = 0; }
                    continue;
                }
                if(open >> i & 1u) mine[i] = key[tid + i * RW_BLOCK];
                mark_odd(odds, i, mine[i] != KEY_EQUAL, mine[i] < KEY_EQUAL);
            }
            __syncthreads();
            sum_odd(odds);
            __syncthreads();
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
                if(mine[i] != KEY_EQUAL) key[odd_before(odds, tid + i * RW_BLOCK) & 0xFFFFu] = mine[i];
            __syncthreads();
            u32 p[RW_ITEMS], deeper[RW_ITEMS];          // position, depth of the member's new group
            u32 go[RW_ITEMS], to_e[RW_ITEMS];           // new slot | first slot of the new group << 16, its end
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
            {
                go[i] = NO_GROUP;
                if((open >> i & 1u) == 0) continue;
                const u32 j = tid + i * RW_BLOCK, s = w.gs[j], e = w.ge[s], d = depth[s];
                p[i] = w.pos[j];
                u32 at, to_s;
                member_place(odds, key, j, s, e, mine[i] != KEY_EQUAL, mine[i] < KEY_EQUAL, mine[i], at, to_s, to_e[i]);
                go[i] = at | to_s << 16;
                const u32 more = shared_by_key(mine[i], reach);
                deeper[i] = to - d < more ? u32(to) : d + more;
            }
            __syncthreads();
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
                if(go[i] != NO_GROUP)
                {
                    const u32 at = go[i] & 0xFFFFu, s = go[i] >> 16;
                    w.pos[at] = p[i];
                    w.gs[at] = u16(s);
                    if(at == s) { w.ge[at] = u16(to_e[i]); depth[at] = deeper[i]; }
                }
            __syncthreads();
            quick -= quick > 0;
        }
        __syncthreads();
        if(tid < RW_WINDOW / 32) w.mask[tid] = 0;
        __syncthreads();
        u32 tied = 0;
        #pragma unroll
        for(int i = 0; i < RW_ITEMS; ++i)
        {
            const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
            if(s == NO_GROUP) continue;
            const u32 x = w.pos[j];
            if(isa) isa[x] = w.head[s];
            if(u32(w.ge[s]) - s < 2)
            {
                if(sa) sa[w.head[j]] = x;
                else
                {
                    u8* const at = sa40 + 5 * u64(w.head[j]);
                    at[0] = u8(x); at[1] = u8(x >> 8); at[2] = u8(x >> 16); at[3] = u8(x >> 24); at[4] = 0;
                }
            }
            else { tied |= 1u << i; atomicOr(&w.mask[j >> 5], 1u << (j & 31)); }
        }
        if(__syncthreads_or(tied != 0))
        {
            const u32 base = window_places(w, &counts->next_small);
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
                if(tied >> i & 1u)
                {
                    const u32 j = tid + i * RW_BLOCK;
                    next[base + w.pre[j >> 5] + __popc(w.mask[j >> 5] & ((1u << (j & 31)) - 1))] = (u64(w.head[w.gs[j]]) << 32) | w.pos[j];
                }
        }
        __syncthreads();
    }
}

constexpr size_t TEXT_SMEM = (sizeof(Window) + 15) / 16 * 16 + size_t(RW_WINDOW) * (8 + 4) + sizeof(Odd_Members);

constexpr int GATHER_UNROLL = 8;
__global__ void __launch_bounds__(256) gather_ranks_kernel(const u64* __restrict__ list, const u64 count, const u32* __restrict__ isa, const u64 n, const u64 h,
                                                          u32* __restrict__ secs)
{
    const u64 first = u64(blockIdx.x) * (256 * GATHER_UNROLL) + threadIdx.x;
    u32 v[GATHER_UNROLL];
    #pragma unroll
    for(int i = 0; i < GATHER_UNROLL; ++i)
    {
        const u64 k = first + u64(i) * 256;
        if(k >= count) continue;
        const u64 x = u64(u32(__ldcs(list + k))) + h;
        v[i] = x < n ? __ldg(isa + x) + u32(MAX_SMALL_H) : u32(n - 1 + h - x);
    }
    #pragma unroll
    for(int i = 0; i < GATHER_UNROLL; ++i)
    {
        const u64 k = first + u64(i) * 256;
        if(k < count) __stcs(secs + k, v[i]);
    }
}

template <typename K>
struct Rank_Window
{
    Group_Starts groups;
    u32 mask[RW_WINDOW / 32];
    u32 pre[RW_WINDOW / 32];
    u32 warp_tot[RW_BLOCK / 32];
    u32 slot;
    K sec[RW_WINDOW];
    Odd_Members odds;
};

template <typename K>
__global__ void __launch_bounds__(RW_BLOCK, 4) refine_by_ranks_kernel(const u64* __restrict__ list, const u64 count, const K* __restrict__ secs, u32* __restrict__ isa,
                                                                     u32* __restrict__ sa, u64* __restrict__ next, Build_Counts* __restrict__ counts)
{
    __shared__ Rank_Window<K> w;
    const u32 tid = threadIdx.x;
    const u64 first = u64(blockIdx.x) * RW_TILE;
    K sec[RW_ITEMS];
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK;
        sec[i] = first + j < count ? __ldcs(secs + first + j) : 0;
        w.sec[j] = sec[i];
    }
    if(tid < RW_WINDOW / 32) w.mask[tid] = 0;
    u64 entry[RW_ITEMS];
    load_entries(w.groups, list, count, first, entry);
    u32 group[RW_ITEMS];        // first slot | end << 16
    u32 odd = 0, smaller = 0;   // a bit per record
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        u32 s, e;
        find_group(w.groups, entry[i], i, s, e);
        group[i] = s | e << 16;
        const K lead = s != NO_GROUP ? w.sec[s] : sec[i];
        odd |= u32(sec[i] != lead) << i;
        smaller |= u32(sec[i] < lead) << i;
        mark_odd(w.odds, i, sec[i] != lead, sec[i] < lead);
    }
    __syncthreads();
    sum_odd(w.odds);
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
        if(odd >> i & 1u) w.sec[odd_before(w.odds, tid + i * RW_BLOCK) & 0xFFFFu] = sec[i];
    __syncthreads();
    u32 place[RW_ITEMS], new_head[RW_ITEMS];        // place: NO_GROUP = not this block's, or alone now
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK, s = group[i] & 0xFFFFu;
        place[i] = NO_GROUP;
        if(s == NO_GROUP) continue;
        u32 at, to_s, to_e;
        member_place(w.odds, w.sec, j, s, group[i] >> 16, (odd >> i & 1u) != 0, (smaller >> i & 1u) != 0, sec[i], at, to_s, to_e);
        const u32 x = u32(entry[i]);
        new_head[i] = u32(entry[i] >> 32) + (to_s - s);
        if(to_s != s) isa[x] = new_head[i];
        if(to_e - to_s == 1) sa[new_head[i]] = x;
        else { place[i] = at; atomicOr(&w.mask[at >> 5], 1u << (at & 31)); }
    }
    const u32 base = window_places(w, &counts->next_small);
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
        if(place[i] != NO_GROUP)
        {
            const u32 q = place[i];
            next[base + w.pre[q >> 5] + __popc(w.mask[q >> 5] & ((1u << (q & 31)) - 1))] = (u64(new_head[i]) << 32) | u32(entry[i]);
        }
}

// ---- groups that follow one another -----------------------------------------------------------------------------------------------
//
// If the suffixes one symbol on from a group's are a whole group again, the two have the same order: the first symbols are the same. In documents that occur
// many times nearly every group has such a follower, up to the next place where the documents differ. So only the groups without one, the ENDS, are ranked by
// doubling, and the others take over the order of the end that their followers lead to. A bit per position says that its suffix's group has a follower; the
// end is as many positions on as there are bits in a row. Some groups, one in 256 by their number, count as ends whatever follows them: no row gets long.
constexpr u32 FORCED_END = 24;      // bits of a group's scrambled number that are 0 in one of 256

// sa[first slot of every group] = its size (the slots are overwritten when their suffixes are known).
__global__ void __launch_bounds__(RW_BLOCK) group_sizes_kernel(const u64* __restrict__ list, const u64 count, u32* __restrict__ sa)
{
    __shared__ Group_Starts groups;
    u64 entry[RW_ITEMS];
    load_entries(groups, list, count, u64(blockIdx.x) * RW_TILE, entry);
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        u32 s, e;
        find_group(groups, entry[i], i, s, e);
        if(s == threadIdx.x + i * RW_BLOCK) sa[u32(entry[i] >> 32)] = e - s;
    }
}

struct Split_Window
{
    Group_Starts groups;
    u32 sec[RW_WINDOW];
    Odd_Members odds;
    u32 keep[RW_WINDOW / 32], keep_before[RW_WINDOW / 32];      // ends: a bit per slot
    u32 keep_slot, passed;
};

// The ends among the list's groups to next (counts->next_small); the bits of the positions whose groups have a follower (counts->large) are set.
// secs: what launch_gather_ranks gives one symbol on.
__global__ void __launch_bounds__(RW_BLOCK, 4) split_followed_kernel(const u64* __restrict__ list, const u64 count, const u32* __restrict__ secs, const u32* __restrict__ sa,
                                                                    u32* __restrict__ bits, u64* __restrict__ next, Build_Counts* __restrict__ counts)
{
    __shared__ Split_Window w;
    const u32 tid = threadIdx.x;
    if(tid == 0) w.passed = 0;          // before load_entries' barriers
    const u64 first = u64(blockIdx.x) * RW_TILE;
    u32 sec[RW_ITEMS];
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK;
        sec[i] = first + j < count ? __ldcs(secs + first + j) : 0;
        w.sec[j] = sec[i];
    }
    u64 entry[RW_ITEMS];
    load_entries(w.groups, list, count, first, entry);
    u32 group[RW_ITEMS];        // first slot | end << 16
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        u32 s, e;
        find_group(w.groups, entry[i], i, s, e);
        group[i] = s | e << 16;
        mark_odd(w.odds, i, s != NO_GROUP && sec[i] != w.sec[s], false);
    }
    __syncthreads();
    sum_odd(w.odds);
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 s = group[i] & 0xFFFFu, e = group[i] >> 16;
        bool followed = false;
        if(s != NO_GROUP && ((odd_before(w.odds, e) ^ odd_before(w.odds, s)) & 0xFFFFu) == 0 && u32(entry[i] >> 32) * 2654435761u >> FORCED_END != 0)
            followed = sec[i] >= MAX_SMALL_H && sa[sec[i] - u32(MAX_SMALL_H)] == e - s;         // the same rank for all of them: a group of several
        if(followed)
        {
            const u32 x = u32(entry[i]);
            atomicOr(bits + (x >> 5), 1u << (x & 31));
        }
        const u32 f = __ballot_sync(0xFFFFFFFFu, followed), k = __ballot_sync(0xFFFFFFFFu, s != NO_GROUP && !followed);
        if(lane_id() == 0)
        {
            if(f) atomicAdd(&w.passed, u32(__popc(f)));
            w.keep[i * (RW_BLOCK / 32) + (tid >> 5)] = k;
        }
    }
    __syncthreads();
    static_assert(RW_WINDOW / 32 == 64, "two words a lane");
    if(tid < 32)
    {
        const u32 k = 2 * lane_id(), a = __popc(w.keep[k]), b = __popc(w.keep[k + 1]), inc = warp_sum(a + b);
        w.keep_before[k] = inc - a - b;
        w.keep_before[k + 1] = inc - b;
        if(lane_id() == 31 && inc) w.keep_slot = atomicAdd(&counts->next_small, inc);
    }
    else if(tid == 32 && w.passed) atomicAdd(&counts->large, w.passed);
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK, word = j >> 5, below = (1u << (j & 31)) - 1;
        if(w.keep[word] >> (j & 31) & 1u) next[u64(w.keep_slot) + w.keep_before[word] + __popc(w.keep[word] & below)] = entry[i];
    }
}

// Bits in a row from position x on (x < n; the bit of the last position is never set).
__device__ __forceinline__ u32 followers(const u64* __restrict__ bits, const u64 x)
{
    u64 word = x >> 6;
    u64 clear = ~__ldg(bits + word) >> (x & 63);
    if(clear) return u32(__ffsll(clear) - 1);
    u32 row = 64 - u32(x & 63);
    while((clear = ~__ldg(bits + ++word)) == 0) row += 64;
    return row + u32(__ffsll(clear) - 1);
}

// secs[i]: what the i-th entry of the list of ends is ordered by, h symbols on: the rank there and, of a suffix whose group has a follower, the rank
// of the end that it leads to: the first is of groups that were told apart before, the second orders inside one of them. A suffix of h symbols comes first.
__global__ void __launch_bounds__(256) gather_pairs_kernel(const u64* __restrict__ list, const u64 count, const u32* __restrict__ isa, const u64 n, const u64 h,
                                                          const u64* __restrict__ bits, u64* __restrict__ secs)
{
    const u64 first = u64(blockIdx.x) * (256 * GATHER_UNROLL) + threadIdx.x;
    u64 v[GATHER_UNROLL];
    #pragma unroll
    for(int i = 0; i < GATHER_UNROLL; ++i)
    {
        const u64 k = first + u64(i) * 256;
        if(k >= count) continue;
        const u64 y = u64(u32(__ldcs(list + k))) + h;
        v[i] = 0;
        if(y >= n) continue;
        const u32 rank = __ldg(isa + y), row = followers(bits, y);
        v[i] = (u64(rank) << 32) | ((row ? __ldg(isa + y + row) : rank) + 1u);
    }
    #pragma unroll
    for(int i = 0; i < GATHER_UNROLL; ++i)
    {
        const u64 k = first + u64(i) * 256;
        if(k < count) __stcs(secs + k, v[i]);
    }
}

// The groups with a follower, once no end is tied: a group leads to the suffixes of one end group, whose ranks by now are its slots, one each. So a suffix is
// as far behind its group's first slot as its end is behind its own. That distance takes the place of the end's rank here (ends: the list of them all as it
// was before any was told apart); the inverse array is then gone through in the text's order, where a suffix and its end are neighbours (Source::FOLLOWED
// below), and sorted into the slots. (With two random reads a suffix in the order of the slots, and the least rank of a group subtracted: 12.9 ms
// for 4e8 near-duplicate suffixes, builds 66.3 ms and 60.5 this way; of 1e8 12.3 and 11.6, of 1e7 to 3e7 the same or less.)
__global__ void __launch_bounds__(256) ends_behind_kernel(const u64* __restrict__ ends, const u64 count, u32* __restrict__ isa, u64* __restrict__ dev_status)
{
    const u64 k = u64(blockIdx.x) * 256 + threadIdx.x;
    if(k >= count) return;
    const u64 e = __ldcs(ends + k);
    const u32 behind = isa[u32(e)] - u32(e >> 32);
    isa[u32(e)] = behind;
    if(behind >= SMALL_GROUP) atomicOr(reinterpret_cast<unsigned long long*>(dev_status), (unsigned long long)CSA_ST_UNSERVED);
}

// ---- lists of groups of any size ----------------------------------------------------------------------------------------------

// A group is small if it has at most SMALL_GROUP members. A block finds the group starts of its tile and of SMALL_GROUP entries on either
// side as bits (as load_entries above), so that a record's group is the stretch between two bits a few words away. Both lists keep the
// order of the records (a group may span many tiles and must stay in one piece): the tiles' counts come first, then their sums
// over the tiles before (size_places_kernel), then the records, 32 side by side. Bound by memory: 4 bytes a record for the counts, 16 for the
// records. (With bisections over the neighbours' heads, one per thread's eight consecutive records, the two passes took 0.61 ms for
// 2^24 records; this way 0.13 ms.)
constexpr int SZ_BLOCK = 256, SZ_TILE = RANK_TILE, SZ_ITEMS = SZ_TILE / SZ_BLOCK, SZ_HALO = int(SMALL_GROUP), SZ_WORDS = (SZ_TILE + 2 * SZ_HALO) / 32;
static_assert(SZ_HALO == SZ_BLOCK && SZ_TILE / 32 == 64, "a warp's words of the window are one halo word, SZ_ITEMS words of the tile and one halo word");

template <bool WRITE>
__global__ void __launch_bounds__(SZ_BLOCK) split_by_size_kernel(const u32* __restrict__ head, const u32* __restrict__ pos, const u64* __restrict__ count_dev,
                                                                u64* __restrict__ next, const u64 cap, uint2* __restrict__ tiles)
{
    __shared__ u32 starts[SZ_WORDS];                // bit j of the window (entry tile + j - SZ_HALO): a group, or what lies behind the list, starts there
    __shared__ int last_in[SZ_TILE / 32], next_in[SZ_TILE / 32];       // of every word of the tile: the start before it and the one behind it, as far as a small group reaches
    __shared__ u32 small_in[SZ_TILE / 32], valid_in[SZ_TILE / 32], before[SZ_TILE / 32];       // per word of the tile; before: small ones | large ones << 16
    __shared__ u32 warp_tot[SZ_BLOCK / 32];
    const u32 tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const u64 tile = u64(blockIdx.x) * SZ_TILE, count = *count_dev;
    if(tile >= count) { if(!WRITE && tid == 0) tiles[blockIdx.x] = make_uint2(0, 0); return; }
    u32 h[SZ_ITEMS + 2], prev[SZ_ITEMS + 2], p[SZ_ITEMS];
    #pragma unroll
    for(int i = 0; i < SZ_ITEMS + 2; ++i)
    {
        const u64 k = tile + i * SZ_BLOCK + tid;        // the entry's index + SZ_HALO
        const bool in = k >= SZ_HALO && k - SZ_HALO < count;
        h[i] = in ? head[k - SZ_HALO] : 0;
        prev[i] = (lane == 0 && in && k > SZ_HALO) ? head[k - SZ_HALO - 1] : 0;
        if(WRITE && i >= 1 && i <= SZ_ITEMS) p[i - 1] = in ? pos[k - SZ_HALO] : 0;
    }
    #pragma unroll
    for(int i = 0; i < SZ_ITEMS + 2; ++i)
    {
        const u64 k = tile + i * SZ_BLOCK + tid;
        const u32 up = __shfl_up_sync(0xFFFFFFFFu, h[i], 1);
        const bool start = k >= SZ_HALO && (k == SZ_HALO || k - SZ_HALO >= count || h[i] != (lane ? up : prev[i]));
        const u32 m = __ballot_sync(0xFFFFFFFFu, start);
        if(lane == 0) starts[i * (SZ_BLOCK / 32) + warp] = m;
    }
    __syncthreads();
    constexpr int REACH = SZ_HALO / 32;
    if(tid < SZ_TILE / 32)
    {
        const int word = REACH + int(tid);
        int last = -int(SMALL_GROUP), next_start = SZ_WORDS * 32 + int(SMALL_GROUP);       // too far away
        #pragma unroll
        for(int k = REACH; k >= 1; --k)
        {
            if(const u32 v = starts[word - k]) last = (word - k) * 32 + 31 - __clz(v);
            if(const u32 v = starts[word + k]) next_start = (word + k) * 32 + __ffs(v) - 1;
        }
        last_in[tid] = last; next_in[tid] = next_start;
    }
    __syncthreads();
    u32 ns = 0, nl = 0;
    #pragma unroll
    for(int i = 0; i < SZ_ITEMS; ++i)
    {
        const int word = REACH + i * (SZ_BLOCK / 32) + int(warp);
        const u32 m = starts[word];
        const int last = last_in[word - REACH], next_start = next_in[word - REACH];
        const u32 upto = m & (0xFFFFFFFFu >> (31 - lane)), behind = m & ~(0xFFFFFFFFu >> (31 - lane));
        const int s = upto ? word * 32 + 31 - __clz(upto) : last, e = behind ? word * 32 + __ffs(behind) - 1 : next_start;
        const bool valid = tile + i * SZ_BLOCK + tid < count;
        const u32 vm = __ballot_sync(0xFFFFFFFFu, valid), sm = __ballot_sync(0xFFFFFFFFu, valid && e - s <= int(SMALL_GROUP));
        ns += __popc(sm); nl += __popc(vm & ~sm);
        if(WRITE && lane == 0) { small_in[i * (SZ_BLOCK / 32) + warp] = sm; valid_in[i * (SZ_BLOCK / 32) + warp] = vm; }
    }
    if(!WRITE)
    {
        if(lane == 0) warp_tot[warp] = ns | nl << 16;
        __syncthreads();
        if(tid == 0)
        {
            u32 all = 0;
            for(int w = 0; w < SZ_BLOCK / 32; ++w) all += warp_tot[w];
            tiles[blockIdx.x] = make_uint2(all & 0xFFFFu, all >> 16);
        }
        return;
    }
    __syncthreads();
    if(tid < 32)            // two words a lane
    {
        const u32 k = 2 * tid;
        const u32 a = __popc(small_in[k]) | __popc(valid_in[k] & ~small_in[k]) << 16, b = __popc(small_in[k + 1]) | __popc(valid_in[k + 1] & ~small_in[k + 1]) << 16;
        const u32 inc = warp_sum(a + b);
        before[k] = inc - a - b;
        before[k + 1] = inc - b;
    }
    __syncthreads();
    const uint2 at = tiles[blockIdx.x];
    #pragma unroll
    for(int i = 0; i < SZ_ITEMS; ++i)
    {
        const u32 word = i * (SZ_BLOCK / 32) + warp, vm = valid_in[word], sm = small_in[word], below = (1u << lane) - 1;
        if((vm >> lane & 1u) == 0) continue;
        const u64 e = (u64(h[i + 1]) << 32) | p[i];
        if(sm >> lane & 1u) next[at.x + (before[word] & 0xFFFFu) + __popc(sm & below)] = e;
        else next[cap - 1 - (at.y + (before[word] >> 16) + __popc(vm & ~sm & below))] = e;
    }
}

// One block: the tiles' counts become their places behind the entries that the two lists hold already, whose lengths are advanced.
__global__ void __launch_bounds__(1024) size_places_kernel(uint2* __restrict__ tiles, const u32 count, Build_Counts* __restrict__ counts)
{
    __shared__ u32 s_s[32], s_l[32];
    __shared__ u32 carry_s, carry_l;
    const u32 tid = threadIdx.x;
    if(tid == 0) { carry_s = counts->next_small; carry_l = counts->large; }
    __syncthreads();
    for(u32 base = 0; base < count; base += 1024)
    {
        const uint2 v = base + tid < count ? tiles[base + tid] : make_uint2(0, 0);
        const u32 is = warp_sum(v.x), il = warp_sum(v.y);
        if(lane_id() == 31) { s_s[tid >> 5] = is; s_l[tid >> 5] = il; }
        __syncthreads();
        u32 ps = carry_s + is - v.x, pl = carry_l + il - v.y;
        for(u32 k = 0; k < (tid >> 5); ++k) { ps += s_s[k]; pl += s_l[k]; }
        if(base + tid < count) tiles[base + tid] = make_uint2(ps, pl);
        __syncthreads();
        if(tid == 1023) { carry_s = ps + v.x; carry_l = pl + v.y; }
        __syncthreads();
    }
    if(tid == 0) { counts->now_small = carry_s - counts->next_small; counts->next_small = carry_s; counts->large = carry_l; }
}

__global__ void unpack_list_kernel(const u64* __restrict__ list, const u64 count, u32* __restrict__ head, u32* __restrict__ pos)
{
    const u64 k = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(k >= count) return;
    const u64 e = list[k];
    head[k] = u32(e >> 32);
    pos[k] = u32(e);
}

// counts->large_depth = the least number of symbols that the suffixes of a group share, over the groups of a list: whole code words among the
// first key_bits bits of their encoding. Only a group's first member is decoded.
__global__ void __launch_bounds__(256) large_depth_kernel(const u64* __restrict__ list, const u64 count, const u16* __restrict__ T, const u64 n, const u32* __restrict__ code,
                                                         const u32 key_bits, Build_Counts* __restrict__ counts)
{
    u32 least = 0xFFFFFFFFu;
    for(u64 k = u64(blockIdx.x) * 256 + threadIdx.x; k < count; k += u64(gridDim.x) * 256)
    {
        const u64 e = __ldg(list + k);
        if(k > 0 && u32(__ldg(list + k - 1) >> 32) == u32(e >> 32)) continue;
        u32 depth = 0, bits = 0;
        for(u64 x = u32(e);; ++x, ++depth)      // a code word has a bit or more
        {
            bits += __ldg(code + (x < n ? u32(T[x]) : 0u)) & 31u;
            if(bits > key_bits) break;
        }
        least = min(least, depth);
    }
    least = __reduce_min_sync(0xFFFFFFFFu, least);
    if(lane_id() == 0 && least != 0xFFFFFFFFu) atomicMin(&counts->large_depth, least);
}

// ---- the inverse array ------------------------------------------------------------------------------------------------------

// (position, rank) pairs of `count` source records into 256 buckets by the top 8 bits of the position. The two sources
// together hold every position once, so bucket b starts at entry b << low_bits and nothing is counted first.
constexpr int MI_BLOCK = 256, MI_ITEMS = 16, MI_TILE = MI_BLOCK * MI_ITEMS;

// Where the pairs come from: the array (`words`), a list, or, the other way round, the inverse array as ends_behind_kernel left it with a bit for every
// position whose group has a follower (`list`): slots and their positions then.
enum class Source { ARRAY, LIST, FOLLOWED };

template <Source FROM>
__device__ __forceinline__ bool inverse_record(const u32* __restrict__ sa, const u64* __restrict__ list, const u64 k, const u64 n, u64& out)
{
    if(FROM == Source::FOLLOWED)
    {
        const u32 row = followers(list, k);
        if(row == 0) return false;
        const u64 slot = u64(__ldg(sa + k)) + __ldg(sa + k + row);
        out = (slot << 32) | u32(k);
        return slot < n;
    }
    if(FROM == Source::ARRAY)
    {
        const u32 x = __ldcs(sa + k);
        out = (u64(x) << 32) | u32(k);
        return x != SA_OPEN;
    }
    const u64 e = __ldcs(list + k);
    out = (e << 32) | (e >> 32);
    return true;
}

template <Source FROM>
__global__ void __launch_bounds__(MI_BLOCK) bucket_ranks_kernel(const u32* __restrict__ sa, const u64* __restrict__ list, const u64 count, const int low_bits,
                                                               u64* __restrict__ out, const u64 out_count, u64* __restrict__ cursor, u64* __restrict__ dev_status)
{
    __shared__ u64 stage[MI_TILE];
    __shared__ u64 base[256];
    __shared__ u32 cnt[256];
    __shared__ u32 warp_tot[8];
    const u32 tid = threadIdx.x;
    const u64 tile_first = u64(blockIdx.x) * MI_TILE;
    cnt[tid] = 0;
    __syncthreads();
    u64 u[MI_ITEMS];
    u32 r[MI_ITEMS];
    #pragma unroll
    for(int k = 0; k < MI_ITEMS; ++k)
    {
        const u64 j = tile_first + tid + k * MI_BLOCK;
        r[k] = 0xFFFFFFFFu;
        if(j < count && inverse_record<FROM>(sa, list, j, out_count, u[k])) r[k] = 0;
    }
    #pragma unroll
    for(int k = 0; k < MI_ITEMS; ++k)
        if(r[k] == 0) r[k] = atomicAdd(&cnt[u32(u[k] >> (32 + low_bits)) & 255u], 1u);
    __syncthreads();
    const u32 c = cnt[tid];
    const u32 inc = warp_sum(c);
    if((tid & 31) == 31) warp_tot[tid >> 5] = inc;
    __syncthreads();
    u32 pre = 0, total = 0;
    #pragma unroll
    for(u32 w = 0; w < 8; ++w) { if(w < (tid >> 5)) pre += warp_tot[w]; total += warp_tot[w]; }
    const u32 start = pre + inc - c;
    if(c) base[tid] = (u64(tid) << low_bits) + atomicAdd(reinterpret_cast<unsigned long long*>(cursor + tid), (unsigned long long)c) - start;
    cnt[tid] = start;
    __syncthreads();
    #pragma unroll
    for(int k = 0; k < MI_ITEMS; ++k)
        if(r[k] != 0xFFFFFFFFu) stage[cnt[u32(u[k] >> (32 + low_bits)) & 255u] + r[k]] = u[k];
    __syncthreads();
    for(u32 j = tid; j < total; j += MI_BLOCK)
    {
        const u64 v = stage[j];
        const u64 at = base[u32(v >> (32 + low_bits)) & 255u] + j;
        if(at < out_count) out[at] = v;
        else atomicOr(reinterpret_cast<unsigned long long*>(dev_status), (unsigned long long)CSA_ST_RANGE);
    }
}

template <Source FROM>
__global__ void __launch_bounds__(256) scatter_ranks_kernel(const u32* __restrict__ sa, const u64* __restrict__ list, const u64 count, const u64 n, u32* __restrict__ to)
{
    const u64 k = u64(blockIdx.x) * 256 + threadIdx.x;
    u64 u;
    if(k < count && inverse_record<FROM>(sa, list, k, n, u)) to[u >> 32] = u32(u);
}

__global__ void __launch_bounds__(256) apply_ranks_kernel(const u64* __restrict__ upd, const u64 count, u32* __restrict__ isa)
{
    const u64 first = (u64(blockIdx.x) * 256 + threadIdx.x) * 2;
    if(first + 1 < count)
    {
        const ulonglong2 v = __ldcs(reinterpret_cast<const ulonglong2*>(upd + first));
        isa[v.x >> 32] = u32(v.x);
        isa[v.y >> 32] = u32(v.y);
    }
    else if(first < count) isa[upd[first] >> 32] = u32(upd[first]);
}

// The same for buckets that are not full: cursor[b] entries in bucket b.
__global__ void __launch_bounds__(256) apply_slots_kernel(const u64* __restrict__ upd, const u64 n, const int low_bits, const u64* __restrict__ cursor, u32* __restrict__ sa)
{
    const u64 first = (u64(blockIdx.x) * 256 + threadIdx.x) * 2;
    if(first >= n) return;
    const u64 filled = __ldg(cursor + (first >> low_bits)), at = first & ((u64(1) << low_bits) - 1);       // a pair lies in one bucket
    if(at + 1 < filled && first + 1 < n)
    {
        const ulonglong2 v = __ldcs(reinterpret_cast<const ulonglong2*>(upd + first));
        sa[v.x >> 32] = u32(v.x);
        sa[v.y >> 32] = u32(v.y);
    }
    else if(at < filled) { const u64 v = upd[first]; sa[v >> 32] = u32(v); }
}

template <Source FROM>
int ranks_from(csa_ctx* ctx, const u32* sa, const u64* list, u64 count, u64 n, u32* to, u64* updates, u64* cursor)
{
    if(count == 0) return CSA_OK;
    const int bits = bits_for(n - 1);
    if(bits <= 24)        // the inverse array stays in L2: straight scatters
        scatter_ranks_kernel<FROM><<<unsigned(div_up(count, 256)), 256, 0, ctx->stream>>>(sa, list, count, n, to);
    else
        bucket_ranks_kernel<FROM><<<unsigned(div_up(count, MI_TILE)), MI_BLOCK, 0, ctx->stream>>>(sa, list, count, bits - 8, updates, n, cursor, ctx->d_status);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

}   // namespace

int read_build_counts(csa_ctx* ctx, u64 most, Build_Counts& c)
{
    CSA_CUDA(ctx, cudaMemcpyAsync(ctx->h_scalars + CSA_COUNTS_WORD, ctx->d_scalars + CSA_COUNTS_WORD, (CSA_STATUS_WORD + 1 - CSA_COUNTS_WORD) * 8, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    CSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if(ctx->h_scalars[CSA_STATUS_WORD] != 0) { u64 b = 0; return csa_sync(ctx, reinterpret_cast<uint64_t*>(&b)); }
    c = *reinterpret_cast<const Build_Counts*>(ctx->h_scalars + CSA_COUNTS_WORD);
    if(c.small > most || u64(c.next_small) + c.large > most) return csa_fail(ctx, CSA_E_DEVICE, "build: the lists of tied suffixes do not add up");
    return CSA_OK;
}

int launch_refine_by_text(csa_ctx* ctx, const u16* T, u64 n, u64 from, u64 to, const u64* list, u64* next, u32* sa, u8* sa40, u32* isa, Build_Counts* counts, u64 expected,
                          u64 most, const u32* code, int key_bits)
{
    to = to < n ? to : n;           // no two suffixes share as much
    CSA_CUDA(ctx, cudaFuncSetAttribute(refine_by_text_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(TEXT_SMEM)));
    const u64 tiles = div_up(expected ? expected : 1, RW_TILE);
    launch_early(refine_by_text_kernel, unsigned(tiles < 148 * 4 ? tiles : 148 * 4), RW_BLOCK, TEXT_SMEM, ctx->stream, T, n, from, to, list, next, sa, sa40, isa, counts, most, code, u32(key_bits));
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_gather_ranks(csa_ctx* ctx, const u64* list, u64 count, const u32* isa, u64 n, u64 h, u32* secs)
{
    if(count == 0) return CSA_OK;
    gather_ranks_kernel<<<unsigned(div_up(count, 256 * GATHER_UNROLL)), 256, 0, ctx->stream>>>(list, count, isa, n, h, secs);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_refine_by_ranks(csa_ctx* ctx, const u64* list, u64 count, const u32* secs, u32* isa, u32* sa, u64* next, Build_Counts* counts)
{
    if(count == 0) return CSA_OK;
    refine_by_ranks_kernel<u32><<<unsigned(div_up(count, RW_TILE)), RW_BLOCK, 0, ctx->stream>>>(list, count, secs, isa, sa, next, counts);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_split_followed(csa_ctx* ctx, const u64* list, u64 count, const u32* isa, u64 n, u32* secs, u32* sa, u32* bits, u64* next, Build_Counts* counts)
{
    if(count == 0) return CSA_OK;
    const unsigned tiles = unsigned(div_up(count, RW_TILE));
    group_sizes_kernel<<<tiles, RW_BLOCK, 0, ctx->stream>>>(list, count, sa);
    CSA_LAUNCH_CHECK(ctx);
    CSA_TRY(launch_gather_ranks(ctx, list, count, isa, n, 1, secs));
    CSA_CUDA(ctx, cudaMemsetAsync(bits, 0, follower_bits_bytes(n), ctx->stream));
    split_followed_kernel<<<tiles, RW_BLOCK, 0, ctx->stream>>>(list, count, secs, sa, bits, next, counts);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_refine_ends(csa_ctx* ctx, const u64* list, u64 count, u64 h, u64* secs, const u32* bits, u32* isa, u64 n, u32* sa, u64* next, Build_Counts* counts)
{
    if(count == 0) return CSA_OK;
    gather_pairs_kernel<<<unsigned(div_up(count, 256 * GATHER_UNROLL)), 256, 0, ctx->stream>>>(list, count, isa, n, h, reinterpret_cast<const u64*>(bits), secs);
    CSA_LAUNCH_CHECK(ctx);
    refine_by_ranks_kernel<u64><<<unsigned(div_up(count, RW_TILE)), RW_BLOCK, 0, ctx->stream>>>(list, count, secs, isa, sa, next, counts);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_place_followed(csa_ctx* ctx, const u64* ends, u64 count, const u32* bits, u32* isa, u64 n, u32* sa, u64* updates)
{
    u64* const cursor = updates + n;
    if(count)
    {
        ends_behind_kernel<<<unsigned(div_up(count, 256)), 256, 0, ctx->stream>>>(ends, count, isa, ctx->d_status);
        CSA_LAUNCH_CHECK(ctx);
    }
    CSA_CUDA(ctx, cudaMemsetAsync(cursor, 0, 256 * 8, ctx->stream));
    CSA_TRY(ranks_from<Source::FOLLOWED>(ctx, isa, reinterpret_cast<const u64*>(bits), n, n, sa, updates, cursor));
    if(bits_for(n - 1) > 24)
    {
        apply_slots_kernel<<<unsigned(div_up(div_up(n, 2), 256)), 256, 0, ctx->stream>>>(updates, n, bits_for(n - 1) - 8, cursor, sa);
        CSA_LAUNCH_CHECK(ctx);
    }
    return CSA_OK;
}

int launch_count_by_size(csa_ctx* ctx, const u32* head, u64 most, const u64* count_dev, Build_Counts* counts, u32* scratch)
{
    if(most == 0) return CSA_OK;
    const unsigned tiles = unsigned(div_up(most, SZ_TILE));
    uint2* const places = reinterpret_cast<uint2*>(scratch);
    split_by_size_kernel<false><<<tiles, SZ_BLOCK, 0, ctx->stream>>>(head, nullptr, count_dev, nullptr, 0, places);
    CSA_LAUNCH_CHECK(ctx);
    size_places_kernel<<<1, 1024, 0, ctx->stream>>>(places, tiles, counts);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_split_by_size(csa_ctx* ctx, const u32* head, const u32* pos, u64 most, const u64* count_dev, u64* next, u64 cap, u32* scratch)
{
    if(most == 0) return CSA_OK;
    split_by_size_kernel<true><<<unsigned(div_up(most, SZ_TILE)), SZ_BLOCK, 0, ctx->stream>>>(head, pos, count_dev, next, cap, reinterpret_cast<uint2*>(scratch));
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_large_depth(csa_ctx* ctx, const u64* list, u64 count, const u16* T, u64 n, const u32* code, int key_bits, Build_Counts* counts)
{
    CSA_CUDA(ctx, cudaMemsetAsync(&counts->large_depth, 0xFF, 4, ctx->stream));
    const u64 blocks = div_up(count, 256);
    large_depth_kernel<<<unsigned(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, ctx->stream>>>(list, count, T, n, code, u32(key_bits), counts);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_unpack_list(csa_ctx* ctx, const u64* list, u64 count, u32* head, u32* pos)
{
    if(count == 0) return CSA_OK;
    unpack_list_kernel<<<unsigned(div_up(count, 256)), 256, 0, ctx->stream>>>(list, count, head, pos);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_make_inverse(csa_ctx* ctx, const u32* sa, u64 n, const u64* small_list, u64 small, const u64* large_list, u64 large, u32* isa, u64* updates)
{
    u64* const cursor = updates + n;
    CSA_CUDA(ctx, cudaMemsetAsync(cursor, 0, 256 * 8, ctx->stream));
    CSA_TRY(ranks_from<Source::ARRAY>(ctx, sa, nullptr, n, n, isa, updates, cursor));
    CSA_TRY(ranks_from<Source::LIST>(ctx, nullptr, small_list, small, n, isa, updates, cursor));
    CSA_TRY(ranks_from<Source::LIST>(ctx, nullptr, large_list, large, n, isa, updates, cursor));
    if(bits_for(n - 1) > 24)
    {
        apply_ranks_kernel<<<unsigned(div_up(div_up(n, 2), 256)), 256, 0, ctx->stream>>>(updates, n, isa);
        CSA_LAUNCH_CHECK(ctx);
    }
    return CSA_OK;
}
