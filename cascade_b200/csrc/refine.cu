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

__device__ __forceinline__ u32 warp_max(u32 v)
{
    #pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const u32 t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if(int(lane_id()) >= o) v = max(v, t);
    }
    return v;
}

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

// A block's window of a list: slot j holds entry first + j. gs[j]: the slot where j's group starts, NO_GROUP where that is not
// inside the block's tile (the group belongs to another block) or past the list's end; ge[gs[j]]: where the group ends.
struct Window
{
    u32 head[RW_WINDOW];
    u32 pos[RW_WINDOW];
    u16 gs[RW_WINDOW];
    u16 ge[RW_WINDOW];
    u32 mask[RW_WINDOW / 32];
    u32 pre[RW_WINDOW / 32];
    u32 warp_tot[RW_BLOCK / 32];
    u32 slot;
};

// Loads the window and finds the groups. A thread's records are the slots tid + i * RW_BLOCK. Ends with a barrier.
__device__ __forceinline__ void load_window(Window& w, const u64* __restrict__ list, const u64 count, const u64 first)
{
    const u32 tid = threadIdx.x;
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK;
        const u64 e = first + j < count ? list[first + j] : ~0ull;      // no group starts at slot 2^32 - 1
        w.head[j] = u32(e >> 32);
        w.pos[j] = u32(e);
    }
    const u32 before = first > 0 ? u32(list[first - 1] >> 32) : 0xFFFFFFFEu;    // another number than any head
    __syncthreads();
    // running last start (as slot + 1, 0 = none) over consecutive slots
    const u32 j0 = tid * RW_ITEMS;
    u32 last = 0, mine[RW_ITEMS];
    u32 prev = j0 > 0 ? w.head[j0 - 1] : before;
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 h = w.head[j0 + i];
        if(h != prev) last = j0 + i + 1;
        mine[i] = last;
        prev = h;
    }
    const u32 inc = warp_max(last);
    if(lane_id() == 31) w.warp_tot[tid >> 5] = inc;
    __syncthreads();
    u32 carry = __shfl_up_sync(0xFFFFFFFFu, inc, 1);
    if(lane_id() == 0) carry = 0;
    for(u32 k = 0; k < (tid >> 5); ++k) carry = max(carry, w.warp_tot[k]);
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 s = max(mine[i], carry);
        w.gs[j0 + i] = (s == 0 || s > RW_TILE || w.head[j0 + i] == 0xFFFFFFFFu) ? u16(NO_GROUP) : u16(s - 1);
    }
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
        if(s != NO_GROUP && (j + 1 == RW_WINDOW || w.gs[j + 1] != s)) w.ge[s] = u16(j + 1);
    }
    __syncthreads();
}

// Appends the slots flagged in w.mask (cleared before, set by atomics, no barrier needed in between) to a list whose length
// *count is advanced; returns the list position of the first. Every thread calls it; the result holds after the call.
__device__ __forceinline__ u32 window_places(Window& w, u32* count)
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

// Orders groups by the symbols [from, to) of their suffixes, eight at a time; the window stays in shared memory over all steps.
// What bounds it is the read of the text: a suffix's symbols are one to five 32-byte sectors in a row.
__global__ void __launch_bounds__(RW_BLOCK) refine_by_text_kernel(const u16* __restrict__ T, const u64 n, const u64 from, const u64 to, const u64* __restrict__ list,
                                                                 u64* __restrict__ next, u32* __restrict__ sa, Build_Counts* __restrict__ counts)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Window& w = *reinterpret_cast<Window*>(smem_raw);
    ulonglong2* const word = reinterpret_cast<ulonglong2*>(smem_raw + (sizeof(Window) + 15) / 16 * 16);     // [RW_WINDOW] the symbols compared in this step
    u8* const split = reinterpret_cast<u8*>(word + RW_WINDOW);      // [RW_WINDOW] by first slot: the group's members differ
    u8* const rest = split + RW_WINDOW;                             // [RW_WINDOW] symbols of the step that the suffix still has, 8 = all
    const u32 tid = threadIdx.x;
    if(counts->oversize != 0) return;           // children still wait for the radix sort: their records lie where `next` would go
    const u64 count = counts->small;
    for(u64 first = u64(blockIdx.x) * RW_TILE; first < count; first += u64(gridDim.x) * RW_TILE)
    {
        load_window(w, list, count, first);
        // from here on head[j] is the suffix-array slot of window slot j, for slots of the block's own groups
        #pragma unroll
        for(int i = 0; i < RW_ITEMS; ++i)
        {
            const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
            if(s != NO_GROUP) w.head[j] += j - s;
        }
        for(u64 d = from; d < to; d += 8)
        {
            bool open = false;
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
            {
                const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
                if(s == NO_GROUP || u32(w.ge[s]) - s < 2) continue;
                open = true;
                const u64 x = u64(w.pos[j]) + d;
                ulonglong2 v = make_ulonglong2(0, 0);
                if(x < n) v = eight_symbols(T, x);
                u64 have = x < n ? n - x : 0;
                u64 want = to - d < 8 ? to - d : 8;
                if(want < 8)        // only the symbols before `to` count
                {
                    if(want <= 4) { v.y = 0; v.x = want == 4 ? v.x : v.x & ~(~0ull >> (16 * want)); }
                    else v.y &= ~(~0ull >> (16 * (want - 4)));
                }
                word[j] = v;
                rest[j] = u8(have < want ? have : want);
                split[j] = 0;
            }
            if(!__syncthreads_or(open)) break;
            bool differs = false;
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
            {
                const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
                if(s == NO_GROUP || u32(w.ge[s]) - s < 2) continue;
                const ulonglong2 a = word[j], b = word[s];
                if(a.x != b.x || a.y != b.y || rest[j] != rest[s]) { split[s] = 1; differs = true; }
            }
            if(!__syncthreads_or(differs)) continue;
            // the members of a group that differs count those before them; then they change places
            u32 p[RW_ITEMS], at[RW_ITEMS], to_s[RW_ITEMS], to_e[RW_ITEMS];
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
            {
                const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
                at[i] = NO_GROUP;
                if(s == NO_GROUP) continue;
                const u32 e = w.ge[s];
                if(e - s < 2 || !split[s]) continue;
                const ulonglong2 a = word[j];
                const u32 ra = rest[j];
                u32 less = 0, eq_before = 0, eq = 0;
                for(u32 k = s; k < e; ++k)
                {
                    const ulonglong2 b = word[k];
                    const u32 rb = rest[k];
                    const bool same_words = b.x == a.x && b.y == a.y;
                    less += (b.x < a.x) || (b.x == a.x && b.y < a.y) || (same_words && rb < ra);
                    const u32 same = same_words && rb == ra;
                    eq += same;
                    eq_before += same && k < j;
                }
                p[i] = w.pos[j];
                to_s[i] = s + less;
                at[i] = s + less + eq_before;
                to_e[i] = s + less + eq;
            }
            __syncthreads();
            #pragma unroll
            for(int i = 0; i < RW_ITEMS; ++i)
                if(at[i] != NO_GROUP)
                {
                    w.pos[at[i]] = p[i];
                    w.gs[at[i]] = u16(to_s[i]);
                    if(at[i] == to_s[i]) w.ge[at[i]] = u16(to_e[i]);
                }
            __syncthreads();
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
            if(u32(w.ge[s]) - s < 2) sa[w.head[j]] = w.pos[j];
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

constexpr size_t TEXT_SMEM = (sizeof(Window) + 15) / 16 * 16 + size_t(RW_WINDOW) * 16 + 2 * RW_WINDOW;

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

__global__ void __launch_bounds__(RW_BLOCK) refine_by_ranks_kernel(const u64* __restrict__ list, const u64 count, const u32* __restrict__ secs, u32* __restrict__ isa,
                                                                  u32* __restrict__ sa, u64* __restrict__ next, Build_Counts* __restrict__ counts)
{
    __shared__ Window w;
    __shared__ u32 sec[RW_WINDOW];
    __shared__ u8 split[RW_WINDOW];
    const u32 tid = threadIdx.x;
    const u64 first = u64(blockIdx.x) * RW_TILE;
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK;
        sec[j] = first + j < count ? secs[first + j] : 0;
        split[j] = 0;
    }
    if(tid < RW_WINDOW / 32) w.mask[tid] = 0;
    load_window(w, list, count, first);
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
        if(s != NO_GROUP && sec[j] != sec[s]) split[s] = 1;
    }
    __syncthreads();
    u32 place[RW_ITEMS], new_head[RW_ITEMS];        // place: NO_GROUP = not this block's, or alone now
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
    {
        const u32 j = tid + i * RW_BLOCK, s = w.gs[j];
        place[i] = NO_GROUP;
        if(s == NO_GROUP) continue;
        const u32 head = w.head[j];
        if(!split[s]) { place[i] = j; new_head[i] = head; }
        else
        {
            const u32 e = w.ge[s], mine = sec[j];
            u32 less = 0, eq_before = 0, eq = 0;
            for(u32 k = s; k < e; ++k)
            {
                const u32 o = sec[k];
                less += o < mine;
                const u32 same = o == mine;
                eq += same;
                eq_before += same && k < j;
            }
            const u32 nh = head + less, x = w.pos[j];
            if(less) isa[x] = nh;
            if(eq == 1) sa[nh] = x;
            else { place[i] = s + less + eq_before; new_head[i] = nh; }
        }
        if(place[i] != NO_GROUP) atomicOr(&w.mask[place[i] >> 5], 1u << (place[i] & 31));
    }
    const u32 base = window_places(w, &counts->next_small);
    #pragma unroll
    for(int i = 0; i < RW_ITEMS; ++i)
        if(place[i] != NO_GROUP)
        {
            const u32 q = place[i];
            next[base + w.pre[q >> 5] + __popc(w.mask[q >> 5] & ((1u << (q & 31)) - 1))] = (u64(new_head[i]) << 32) | w.pos[tid + i * RW_BLOCK];
        }
}

// ---- lists of groups of any size ----------------------------------------------------------------------------------------------

// A group is small if it has at most SMALL_GROUP members, which a look at the SMALL_GROUP entries before and behind a record tells.
// Both lists keep the order of the records (a group may span many tiles and must stay in one piece): the tiles' counts come
// first, then their sums over the tiles before (size_places_kernel), then the records.
constexpr int SZ_BLOCK = 256, SZ_ITEMS = RANK_TILE / SZ_BLOCK, SZ_TILE = SZ_BLOCK * SZ_ITEMS, SZ_WINDOW = SZ_TILE + 2 * int(SMALL_GROUP);

template <bool WRITE>
__global__ void __launch_bounds__(SZ_BLOCK) split_by_size_kernel(const u32* __restrict__ head, const u32* __restrict__ pos, const u64* __restrict__ count_dev,
                                                                u64* __restrict__ next, const u64 cap, uint2* __restrict__ tiles)
{
    __shared__ u32 h[SZ_WINDOW];
    __shared__ u32 warp_s[SZ_BLOCK / 32], warp_l[SZ_BLOCK / 32];
    const u32 tid = threadIdx.x;
    const u64 tile = u64(blockIdx.x) * SZ_TILE, count = *count_dev;
    if(tile >= count) { if(!WRITE && tid == 0) tiles[blockIdx.x] = make_uint2(0, 0); return; }
    for(u32 j = tid; j < u32(SZ_WINDOW); j += SZ_BLOCK)
    {
        const u64 k = tile + j;             // entry k - SMALL_GROUP
        h[j] = (k >= SMALL_GROUP && k - SMALL_GROUP < count) ? head[k - SMALL_GROUP] : 0xFFFFFFFFu;
    }
    __syncthreads();
    u32 kind[SZ_ITEMS], ns = 0, nl = 0;     // a thread's records are consecutive
    #pragma unroll
    for(int i = 0; i < SZ_ITEMS; ++i)
    {
        const u32 j = SMALL_GROUP + tid * SZ_ITEMS + i;
        kind[i] = 0;
        if(tile + tid * SZ_ITEMS + i >= count) continue;
        const u32 me = h[j];
        u32 a = 0, b = SMALL_GROUP;         // members before me, as far as SMALL_GROUP
        while(a < b) { const u32 m = (a + b + 1) >> 1; if(h[j - m] == me) a = m; else b = m - 1; }
        u32 c = 0, d = SMALL_GROUP;         // members behind me
        while(c < d) { const u32 m = (c + d + 1) >> 1; if(h[j + m] == me) c = m; else d = m - 1; }
        const bool small = a + c + 1 <= SMALL_GROUP;
        kind[i] = small ? 1 : 2;
        ns += small; nl += !small;
    }
    const u32 is = warp_sum(ns), il = warp_sum(nl);
    if(lane_id() == 31) { warp_s[tid >> 5] = is; warp_l[tid >> 5] = il; }
    __syncthreads();
    u32 ps = is - ns, pl = il - nl;
    for(u32 k = 0; k < (tid >> 5); ++k) { ps += warp_s[k]; pl += warp_l[k]; }
    if(!WRITE)
    {
        if(tid == SZ_BLOCK - 1) tiles[blockIdx.x] = make_uint2(ps + ns, pl + nl);
        return;
    }
    const uint2 at = tiles[blockIdx.x];
    ps += at.x; pl += at.y;
    #pragma unroll
    for(int i = 0; i < SZ_ITEMS; ++i)
    {
        if(kind[i] == 0) continue;
        const u64 k = tile + tid * SZ_ITEMS + i;
        const u64 e = (u64(h[SMALL_GROUP + tid * SZ_ITEMS + i]) << 32) | pos[k];
        if(kind[i] == 1) next[ps++] = e;
        else next[cap - 1 - pl++] = e;
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
    if(tid == 0) { counts->next_small = carry_s; counts->large = carry_l; }
}

__global__ void unpack_list_kernel(const u64* __restrict__ list, const u64 count, u32* __restrict__ head, u32* __restrict__ pos)
{
    const u64 k = u64(blockIdx.x) * blockDim.x + threadIdx.x;
    if(k >= count) return;
    const u64 e = list[k];
    head[k] = u32(e >> 32);
    pos[k] = u32(e);
}

// ---- the inverse array ------------------------------------------------------------------------------------------------------

// (position, rank) pairs of `count` source records into 256 buckets by the top 8 bits of the position. The two sources
// together hold every position once, so bucket b starts at entry b << low_bits and nothing is counted first.
constexpr int MI_BLOCK = 256, MI_ITEMS = 16, MI_TILE = MI_BLOCK * MI_ITEMS;

template <bool FROM_SA>
__device__ __forceinline__ bool inverse_record(const u32* __restrict__ sa, const u64* __restrict__ list, const u64 k, u64& out)
{
    if(FROM_SA)
    {
        const u32 x = __ldcs(sa + k);
        out = (u64(x) << 32) | u32(k);
        return x != SA_OPEN;
    }
    const u64 e = __ldcs(list + k);
    out = (e << 32) | (e >> 32);
    return true;
}

template <bool FROM_SA>
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
        if(j < count && inverse_record<FROM_SA>(sa, list, j, u[k])) r[k] = 0;
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

template <bool FROM_SA>
__global__ void __launch_bounds__(256) scatter_ranks_kernel(const u32* __restrict__ sa, const u64* __restrict__ list, const u64 count, u32* __restrict__ isa)
{
    const u64 k = u64(blockIdx.x) * 256 + threadIdx.x;
    u64 u;
    if(k < count && inverse_record<FROM_SA>(sa, list, k, u)) isa[u >> 32] = u32(u);
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

template <bool FROM_SA>
int ranks_from(csa_ctx* ctx, const u32* sa, const u64* list, u64 count, u64 n, u32* isa, u64* updates, u64* cursor)
{
    if(count == 0) return CSA_OK;
    const int bits = bits_for(n - 1);
    if(bits <= 24)        // the inverse array stays in L2: straight scatters
        scatter_ranks_kernel<FROM_SA><<<unsigned(div_up(count, 256)), 256, 0, ctx->stream>>>(sa, list, count, isa);
    else
        bucket_ranks_kernel<FROM_SA><<<unsigned(div_up(count, MI_TILE)), MI_BLOCK, 0, ctx->stream>>>(sa, list, count, bits - 8, updates, n, cursor, ctx->d_status);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

}   // namespace

int launch_refine_by_text(csa_ctx* ctx, const u16* T, u64 n, u64 from, u64 to, const u64* list, u64* next, u32* sa, Build_Counts* counts, u64 expected)
{
    CSA_CUDA(ctx, cudaFuncSetAttribute(refine_by_text_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(TEXT_SMEM)));
    const u64 tiles = div_up(expected ? expected : 1, RW_TILE);
    refine_by_text_kernel<<<unsigned(tiles < 148 * 3 ? tiles : 148 * 3), RW_BLOCK, TEXT_SMEM, ctx->stream>>>(T, n, from, to, list, next, sa, counts);
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
    refine_by_ranks_kernel<<<unsigned(div_up(count, RW_TILE)), RW_BLOCK, 0, ctx->stream>>>(list, count, secs, isa, sa, next, counts);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_split_by_size(csa_ctx* ctx, const u32* head, const u32* pos, u64 most, const u64* count_dev, u64* next, u64 cap, Build_Counts* counts, u32* scratch)
{
    if(most == 0) return CSA_OK;
    const unsigned tiles = unsigned(div_up(most, SZ_TILE));
    uint2* const places = reinterpret_cast<uint2*>(scratch);
    split_by_size_kernel<false><<<tiles, SZ_BLOCK, 0, ctx->stream>>>(head, pos, count_dev, next, cap, places);
    CSA_LAUNCH_CHECK(ctx);
    size_places_kernel<<<1, 1024, 0, ctx->stream>>>(places, tiles, counts);
    CSA_LAUNCH_CHECK(ctx);
    split_by_size_kernel<true><<<tiles, SZ_BLOCK, 0, ctx->stream>>>(head, pos, count_dev, next, cap, places);
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
    CSA_TRY(ranks_from<true>(ctx, sa, nullptr, n, n, isa, updates, cursor));
    CSA_TRY(ranks_from<false>(ctx, nullptr, small_list, small, n, isa, updates, cursor));
    CSA_TRY(ranks_from<false>(ctx, nullptr, large_list, large, n, isa, updates, cursor));
    if(bits_for(n - 1) > 24)
    {
        apply_ranks_kernel<<<unsigned(div_up(div_up(n, 2), 256)), 256, 0, ctx->stream>>>(updates, n, isa);
        CSA_LAUNCH_CHECK(ctx);
    }
    return CSA_OK;
}
