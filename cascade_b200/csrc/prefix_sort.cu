// Generation 0 of the resident build: the suffixes sorted by the first bits of their ENCODED symbols.
//
// Token ids are far from uniform: of the 16 bits of a symbol a Zipf text fills about 9.4, so a radix sort of raw symbols
// spends nearly half of its digit passes on bits that say nothing, and four raw symbols (64 bits) still leave 30 % of the
// suffixes of a 2e9-token text tied. Here the symbols are first given an order-preserving prefix code made from a sample of the
// text (a weight-balanced binary tree over the 65536 symbols in numeric order: within 0.1 bit of the entropy on Zipf
// text). Encoded suffixes have nearly uniform bits, which pays four times:
//   * 42 bits tell 2e9 suffixes apart but for a few in a thousand (they cover about 4.4 symbols);
//   * a record is 8 bytes, 32 key bits + 32 position bits, as the bits of the first split need not be kept;
//   * a split by the TOP bits makes evenly filled buckets, so it needs no sampling of splitters, and as its order inside
//     a bucket is free it needs no stable ranking and no look-back: two unordered splits of up to 10 + 11 bits leave buckets
//     ("children") of about 2000 suffixes;
//   * inside a child the keys are so even that a record's place follows from its key by interpolation, give or take a record
//     or two: one block finishes a run of children in shared memory.
// So a suffix is moved three times (two splits, one local sort) where a least-significant-digit sort of 64 bits moves it eight
// times. Any text is sorted correctly; what an uneven text (one symbol repeated, a few symbols in a pattern) changes is only
// how many children do not fit a block and go through the radix sort instead.
//
// It stands for select_pivots, partition and the sort of initial_rank (src/GPU_SACA.cu:290-364, 737-826, 1111-1331).
#include "prefix_sort.cuh"

#include <algorithm>
#include <atomic>

namespace
{

constexpr int TEXT_ITEMS = 16;              // consecutive symbols per thread of an encoding block
constexpr int LOOKAHEAD = 64;               // a key of up to 64 bits needs at most 64 symbols
constexpr int MAX_B1 = 10, MAX_B2 = 11;
constexpr int SPLIT_ITEMS = 16;             // records per thread of the second split
// Threads of its blocks. Where a parent has 1024 children a tile of 16384 records writes runs of 16 of them and one of 8192 only 8: a build of 2e9 tokens 36.8 ms by blocks of 1024 threads, 38.0 by 512,
// 1e9 18.3 and 18.9. With 512 children the smaller blocks, two to an SM, are 1 to 2 % faster (5e8: 8.84 and 9.00 ms).
inline int split_block(const int b2) { return b2 >= 10 ? 1024 : 512; }
constexpr u32 SORT_BLOCKS = 3;               // of the local sort an SM
constexpr u32 MEDIUM_CAP = 512 * 16;        // records of the largest child that a block holds

// ---- the code ----------------------------------------------------------------------------------------------------------------

constexpr int HIST_BLOCK = 1024;
constexpr size_t HIST_SMEM = 65536 * 2;

// Symbol counts of `vectors` pieces of 8 symbols spread evenly over the text (all pieces where vectors = whole pieces of the
// text; the last n % 8 symbols are then counted too). A block counts in shared memory, two 16-bit counters a word: it takes
// fewer than 65536 symbols.
__global__ void __launch_bounds__(HIST_BLOCK) sample_symbols_kernel(const u16* __restrict__ T, const u64 n, const u64 vectors, u32* __restrict__ hist)
{
    let_next_in();
    extern __shared__ __align__(16) u32 h[];
    for(u32 i = threadIdx.x; i < 32768; i += HIST_BLOCK) h[i] = 0;
    __syncthreads();
    const u64 pieces = n / 8;
    for(u64 v = u64(blockIdx.x) * HIST_BLOCK + threadIdx.x; v < vectors; v += u64(gridDim.x) * HIST_BLOCK)
    {
        // one piece of every stretch, at a place of its own: a text of records of one length would meet an even step at the same few places of
        // every record (2^24 tokens, sixteen documents of 2048 copied over and over: 11.4 ms a build, this way 9.6 ms)
        const u64 at = vectors == pieces ? v : (v * pieces + (u64(u32(v) * 2654435769u) * pieces >> 32)) / vectors;
        const uint4 q = reinterpret_cast<const uint4*>(T)[at];
        const u32 w[4] = {q.x, q.y, q.z, q.w};
        #pragma unroll
        for(int k = 0; k < 4; ++k)
        {
            const u32 a = w[k] & 0xFFFFu, b = w[k] >> 16;
            atomicAdd(&h[a >> 1], (a & 1) ? 0x10000u : 1u);
            atomicAdd(&h[b >> 1], (b & 1) ? 0x10000u : 1u);
        }
    }
    if(blockIdx.x == 0 && vectors == pieces && threadIdx.x < n % 8)
    {
        const u32 a = T[pieces * 8 + threadIdx.x];
        atomicAdd(&h[a >> 1], (a & 1) ? 0x10000u : 1u);
    }
    __syncthreads();
    for(u32 i = threadIdx.x; i < 32768; i += HIST_BLOCK)
    {
        const u32 c = h[i];
        if(c & 0xFFFFu) atomicAdd(&hist[2 * i], c & 0xFFFFu);
        if(c >> 16) atomicAdd(&hist[2 * i + 1], c >> 16);
    }
}

__device__ __forceinline__ u32 warp_inclusive(u32 v)
{
    #pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const u32 t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if(int(lane_id()) >= o) v += t;
    }
    return v;
}

// Exclusive sum over the block's threads; every thread calls it. warp_tot: BLOCK / 32 words. Returns the exclusive sum, and the
// total in `total`. Ends with a barrier.
template <int BLOCK>
__device__ __forceinline__ u32 block_exclusive(const u32 v, u32* warp_tot, u32& total)
{
    const u32 inc = warp_inclusive(v);
    if(lane_id() == 31) warp_tot[threadIdx.x >> 5] = inc;
    __syncthreads();
    const u32 t = lane_id() < BLOCK / 32 ? warp_tot[lane_id()] : 0;        // every warp sums the warps' totals
    const u32 upto = warp_inclusive(t);
    const u32 all = __shfl_sync(0xFFFFFFFFu, upto, 31), pre = __shfl_sync(0xFFFFFFFFu, upto - t, threadIdx.x >> 5);
    __syncthreads();
    total = all;
    return pre + inc - v;
}

// Weights and code words in one launch. Every block holds the prefix sums of all 65536 weights in shared memory, 24 bits each (16
// and 8 apart), and gives CODE_WALKERS symbols their words; the weights are scale * count + 1 (every symbol must have a code word:
// the sample may have missed it), below 2^23 together. COUNT: the text is short, and every block counts its symbols by itself.
//
// One symbol per thread walks down the tree: a node is a range of symbols, split where the weights of its halves come closest,
// but never so that a half has more symbols than code words are left for it. All symbols of a node find the same split. The walk
// is one chain of some 150 dependent reads, which is why the sums lie in shared memory: with the sums made by one block and read
// through L2, the two launches took 98 us of a short build's 190.
constexpr int CODE_BLOCK = 1024;
constexpr u32 CODE_WALKERS = 512;               // threads of a block that walk: more warps would wait for shared memory, not for its latency
constexpr u64 CODE_COUNT_MAX = 1 << 14;         // longest text that every block counts by itself (16-bit counters)
constexpr u32 CODE_LOW_BYTES = (65536 + 8) * 2;
constexpr size_t CODE_SMEM = CODE_LOW_BYTES + 65536 + 8;

template <bool COUNT>
__global__ void __launch_bounds__(CODE_BLOCK) make_code_kernel(const u16* __restrict__ T, const u32 n, const u32* __restrict__ hist, const u32 scale, u32* __restrict__ code,
                                                              u32* __restrict__ cnt1, u32* __restrict__ counts, u32* __restrict__ cnt2, const u32 children)
{
    let_next_in();
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u16* const low = reinterpret_cast<u16*>(smem_raw);
    u8* const high = smem_raw + CODE_LOW_BYTES;
    __shared__ u32 warp_tot[CODE_BLOCK / 32];
    const u32 tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    if(blockIdx.x == 0)         // the counters that the kernels behind this one start from
    {
        cnt1[tid] = 0;
        if(tid < sizeof(Build_Counts) / 4) counts[tid] = 0;
    }
    for(u32 i = blockIdx.x * CODE_BLOCK + tid; i < children; i += gridDim.x * CODE_BLOCK) cnt2[i] = 0;
    if(COUNT)
    {
        for(u32 i = tid; i < 65536 * 2 / 16; i += CODE_BLOCK) reinterpret_cast<uint4*>(low)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        for(u32 i = tid; i < n; i += CODE_BLOCK)
        {
            const u32 a = T[i];
            atomicAdd(reinterpret_cast<u32*>(low) + (a >> 1), (a & 1) ? 0x10000u : 1u);
        }
        __syncthreads();
    }
    // a warp takes 2048 consecutive symbols, 128 at a time: their sum, then their prefix sums behind those of the warps before
    auto counts_of = [&](const u32 s) -> uint4
    {
        if(!COUNT) return __ldg(reinterpret_cast<const uint4*>(hist + s));
        const ushort4 v = *reinterpret_cast<const ushort4*>(low + s);
        return make_uint4(v.x, v.y, v.z, v.w);
    };
    u32 mine = 0;
    #pragma unroll
    for(int k = 0; k < 16; ++k)
    {
        const uint4 c = counts_of(warp * 2048 + k * 128 + lane * 4);
        mine += c.x + c.y + c.z + c.w;
    }
    mine = scale * __reduce_add_sync(0xFFFFFFFFu, mine) + 2048;
    if(lane == 0) warp_tot[warp] = mine;
    __syncthreads();
    {
        u32 run = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? warp_tot[lane] : 0u);
        #pragma unroll 8
        for(int k = 0; k < 16; ++k)
        {
            const u32 s = warp * 2048 + k * 128 + lane * 4;
            const uint4 c = counts_of(s);
            const u32 sum = scale * (c.x + c.y + c.z + c.w) + 4, inc = warp_inclusive(sum);
            const u32 x = run + inc - sum, y = x + scale * c.x + 1, z = y + scale * c.y + 1, w = z + scale * c.z + 1;
            *reinterpret_cast<uint2*>(low + s) = make_uint2(__byte_perm(x, y, 0x5410), __byte_perm(z, w, 0x5410));
            *reinterpret_cast<u32*>(high + s) = __byte_perm(__byte_perm(x, y, 0x0062), __byte_perm(z, w, 0x0062), 0x5410);
            run += __shfl_sync(0xFFFFFFFFu, inc, 31);
        }
        if(tid == CODE_BLOCK - 1) { low[65536] = u16(run); high[65536] = u8(run >> 16); }
    }
    __syncthreads();
    auto prefix = [&](const u32 m) { return u32(low[m]) | u32(high[m]) << 16; };

    if(tid >= CODE_WALKERS) return;
    const u32 s = blockIdx.x * CODE_WALKERS + tid, s_first = s - lane;
    u32 lo = 0, hi = 65536, word = 0;
    int left = CODE_MAX_LEN;            // bits left below the node
    u32 plo = 0, phi = prefix(65536);
    // The split of a node from the first boundary at or past the middle.
    auto settle = [&](u32& m, u32& pm, const u32 twice_mid)
    {
        if(m > lo + 1)
        {
            const u32 pb = prefix(m - 1);
            if(2 * pm >= twice_mid && twice_mid - 2 * pb <= 2 * pm - twice_mid) { --m; pm = pb; }
        }
        const u32 room = 1u << (left - 1);
        if(m - lo > room) { m = lo + room; pm = prefix(m); }
        else if(hi - m > room) { m = hi - room; pm = prefix(m); }
        --left;
    };
    auto descend = [&](const u32 m, const u32 pm)
    {
        if(s < m) { hi = m; phi = pm; }
        else { lo = m; plo = pm; word |= 1u << (31 - (CODE_MAX_LEN - 1 - left)); }
    };
    // As long as a warp's symbols are in one node, all lanes look for its split: 32 boundaries at a time.
    bool together = true;
    while(together && hi - lo > 1)
    {
        const u32 twice_mid = plo + phi;
        u32 a = lo + 1, b = hi - 1;     // the split: kept inside (lo, hi)
        while(a < b)
        {
            const u32 step = b - a <= 32 ? 1 : (b - a + 32) / 33, probe = a + (lane + 1) * step - 1;
            const u32 before = __popc(__ballot_sync(0xFFFFFFFFu, probe < b && 2 * prefix(probe) < twice_mid));     // a leading run of lanes
            if(before < 32) b = min(b, a + (before + 1) * step - 1);
            a += before * step;
        }
        u32 m = a, pm = prefix(m);
        settle(m, pm, twice_mid);
        together = m <= s_first || m > s_first + 31;
        descend(m, pm);
    }
    while(hi - lo > 1)
    {
        const u32 twice_mid = plo + phi;
        u32 a = lo + 1, b = hi - 1;
        while(a < b)
        {
            const u32 m = (a + b) >> 1;
            if(2 * prefix(m) >= twice_mid) b = m; else a = m + 1;
        }
        u32 m = a, pm = prefix(m);
        settle(m, pm, twice_mid);
        descend(m, pm);
    }
    code[s] = word | u32(CODE_MAX_LEN - left);
}

// ---- encoding a tile of the text ------------------------------------------------------------------------------------------------

// A block of BLOCK threads takes BLOCK * TEXT_ITEMS consecutive symbols, of which the last LOOKAHEAD only complete the keys of
// those before them: a tile yields the keys of TILE_POSITIONS suffixes.
template <int BLOCK> constexpr int TILE_POSITIONS = BLOCK * TEXT_ITEMS - LOOKAHEAD;

// The first 64 bits of a suffix's encoding follow from those of the next suffix: its own symbol's code word, then the other's bits.
// So a thread walks its symbols from the last to the first with one 64-bit window, and needs only the window behind its last symbol.
__device__ __forceinline__ u64 before(const u32 entry, const u64 window) { return u64(entry & ~31u) << 32 | window >> (entry & 31u); }

template <int BLOCK> struct Tile_Code
{
    u64 window[BLOCK];      // of every thread: the first bits of its symbols
    u32 bits[BLOCK];        // and how many its symbols have
};

// The code entries of the thread's symbols [first + threadIdx.x * TEXT_ITEMS, + TEXT_ITEMS) in ent, and the window behind the last. Symbols
// past the text's end count as 0. first is a multiple of 16 and T is 16-byte aligned with CSA_TEXT_PAD readable symbols behind n.
// The windows of the last LOOKAHEAD symbols' threads are not complete. Ends without a barrier behind the reads of `tc`.
// (Writing the code words one behind the other into shared memory and reading every suffix's words from there, the scatter at 2e9 symbols
// took 12.9 ms, at 88 % of L1's wavefronts; this way 10.7 ms.)
template <int BLOCK>
__device__ __forceinline__ u64 encode_tile(const u16* __restrict__ T, const u64 n, const u64 first, const u32* __restrict__ code, Tile_Code<BLOCK>& tc, u32 (&ent)[TEXT_ITEMS])
{
    const u64 at = first + u64(threadIdx.x) * TEXT_ITEMS;
    u32 sym2[TEXT_ITEMS / 2];
    if(at + TEXT_ITEMS <= n + CSA_TEXT_PAD)
    {
        const uint4 a = *reinterpret_cast<const uint4*>(T + at), b = *reinterpret_cast<const uint4*>(T + at + 8);
        sym2[0] = a.x; sym2[1] = a.y; sym2[2] = a.z; sym2[3] = a.w;
        sym2[4] = b.x; sym2[5] = b.y; sym2[6] = b.z; sym2[7] = b.w;
    }
    else
    {
        #pragma unroll
        for(int i = 0; i < TEXT_ITEMS / 2; ++i)
            sym2[i] = (at + 2 * i < n ? u32(T[at + 2 * i]) : 0u) | (at + 2 * i + 1 < n ? u32(T[at + 2 * i + 1]) << 16 : 0u);
    }
    #pragma unroll
    for(int i = 0; i < TEXT_ITEMS; ++i) ent[i] = __ldg(code + ((i & 1) ? sym2[i >> 1] >> 16 : sym2[i >> 1] & 0xFFFFu));
    u64 own = 0;
    u32 bits = 0;
    #pragma unroll
    for(int i = TEXT_ITEMS - 1; i >= 0; --i) { own = before(ent[i], own); bits += ent[i] & 31u; }
    tc.window[threadIdx.x] = own;
    tc.bits[threadIdx.x] = bits;
    __syncthreads();
    u64 behind = 0;
    u32 have = 0;       // a thread's symbols have 16 bits or more: four threads fill a window, one as a rule
    for(u32 t = threadIdx.x + 1; t < BLOCK && have < 64; ++t) { behind |= tc.window[t] >> have; have += tc.bits[t]; }
    return behind;
}

// ---- first split: by the top bits, straight from the text -----------------------------------------------------------------------

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) count_text_kernel(const u16* __restrict__ T, const u64 n, const u32* __restrict__ code, const int bits, u32* __restrict__ counts)
{
    let_next_in();
    wait_for_previous();
    __shared__ Tile_Code<BLOCK> tc;
    __shared__ u32 cnt[1 << MAX_B1];
    const u32 bins = 1u << bits;
    for(u32 i = threadIdx.x; i < bins; i += BLOCK) cnt[i] = 0;
    const u64 first = u64(blockIdx.x) * TILE_POSITIONS<BLOCK>;
    u32 ent[TEXT_ITEMS];
    u64 window = encode_tile<BLOCK>(T, n, first, code, tc, ent);
    const u32 local = threadIdx.x * TEXT_ITEMS;
    const u64 room = n - first;
    const u32 valid = room < u64(TILE_POSITIONS<BLOCK>) ? u32(room) : u32(TILE_POSITIONS<BLOCK>);
    #pragma unroll
    for(int i = TEXT_ITEMS - 1; i >= 0; --i)
    {
        window = before(ent[i], window);
        if(local + i < valid) atomicAdd(&cnt[u32(window >> 32) >> (32 - bits)], 1u);
    }
    __syncthreads();
    for(u32 i = threadIdx.x; i < bins; i += BLOCK)
        if(cnt[i]) atomicAdd(&counts[i], cnt[i]);
}

// The same for long texts: one block an SM holds the whole code in shared memory, cut to what the first split looks at (12 bits
// of the code word and a length up to 15: 16 bits a symbol), since a gather from the 256 KB table through L1 is what bounds the
// kernel above (5.5 ms at 2e9 symbols, this way 1.7 ms). A warp goes through strips of 512 symbols by itself; the last lane's 16
// only complete the windows before them.
constexpr int COUNT_BLOCK = 1024;
constexpr u32 STRIP = 31 * TEXT_ITEMS;
constexpr size_t COUNT_SMEM = 65536 * 2;
static_assert(MAX_B1 <= 12 && TEXT_ITEMS >= 12, "12 bits of a code word are kept, and the next lane's symbols have as many");

__global__ void __launch_bounds__(COUNT_BLOCK) count_long_text_kernel(const u16* __restrict__ T, const u64 n, const u32* __restrict__ code, const int bits, u32* __restrict__ counts)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u16* const table = reinterpret_cast<u16*>(smem_raw);
    __shared__ u32 cnt[1 << MAX_B1];
    const u32 bins = 1u << bits, lane = lane_id();
    for(u32 i = threadIdx.x; i < bins; i += COUNT_BLOCK) cnt[i] = 0;
    for(u32 i = threadIdx.x; i < 65536 / 4; i += COUNT_BLOCK)
    {
        const uint4 c = __ldg(reinterpret_cast<const uint4*>(code) + i);
        auto cut = [](const u32 e) { return u16((e >> 16 & 0xFFF0u) | min(e & 31u, 15u)); };
        reinterpret_cast<ushort4*>(table)[i] = make_ushort4(cut(c.x), cut(c.y), cut(c.z), cut(c.w));
    }
    __syncthreads();
    const u64 strips = (n + STRIP - 1) / STRIP, step = u64(gridDim.x) * (COUNT_BLOCK / 32);
    u64 strip = u64(blockIdx.x) * (COUNT_BLOCK / 32) + (threadIdx.x >> 5);
    auto load = [&](const u64 s, uint4& a, uint4& b)
    {
        const u64 at = s * STRIP + lane * TEXT_ITEMS;
        a = make_uint4(0, 0, 0, 0); b = a;
        if(s < strips && at + TEXT_ITEMS <= n + CSA_TEXT_PAD)       // what is cut off lies past the text and counts as 0
        {
            a = *reinterpret_cast<const uint4*>(T + at);
            b = *reinterpret_cast<const uint4*>(T + at + 8);
        }
    };
    uint4 a, b;
    load(strip, a, b);
    for(; strip < strips; strip += step)
    {
        const u32 sym2[TEXT_ITEMS / 2] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        load(strip + step, a, b);
        u32 ent[TEXT_ITEMS];
        #pragma unroll
        for(int i = 0; i < TEXT_ITEMS; ++i) ent[i] = table[(i & 1) ? sym2[i >> 1] >> 16 : sym2[i >> 1] & 0xFFFFu];
        auto step_back = [](const u32 e, const u32 w) { return (e & 0xFFF0u) << 16 | w >> (e & 15u); };
        u32 own = 0;
        #pragma unroll
        for(int i = 11; i >= 0; --i) own = step_back(ent[i], own);     // 12 symbols have 12 bits or more
        u32 window = __shfl_down_sync(0xFFFFFFFFu, own, 1);
        const u64 at = strip * STRIP + lane * TEXT_ITEMS;
        const u32 valid = lane == 31 || at >= n ? 0u : (n - at < TEXT_ITEMS ? u32(n - at) : u32(TEXT_ITEMS));
        #pragma unroll
        for(int i = TEXT_ITEMS - 1; i >= 0; --i)
        {
            window = step_back(ent[i], window);
            if(u32(i) < valid) atomicAdd(&cnt[window >> (32 - bits)], 1u);
        }
    }
    __syncthreads();
    for(u32 i = threadIdx.x; i < bins; i += COUNT_BLOCK)
        if(cnt[i]) atomicAdd(&counts[i], cnt[i]);
}

// The batches of one parent, by a block of 1024 threads: off (shared memory, a barrier behind its writes) holds where its children start and where they end, from 0. A batch is a run of
// children of one segment with up to `most` records, no longer than longest_run, or a single child (batch_end); its entry: the first slot, the records, the children (children_entry). A child of more than SORT_MOST goes to
// one of the other lists. only: there is no other parent. The batches of a segment follow from one another, so a thread forms them; bisecting and writing are side by side.
// A run of children of one parent in one word: there are up to 2^21 children, and 2^MAX_B2 of a parent.
static_assert(MAX_B1 + 2 * MAX_B2 <= 32, "an entry is a word");
__device__ __forceinline__ u32 children_entry(const u32 first, const u32 count) { return first << MAX_B2 | (count - 1); }

struct Batch_Room { u32 used, at; u16 next[1 << MAX_B2]; u32 heads[(1 << MAX_B2) / 32]; };
__device__ __forceinline__ void form_batches(Batch_Room& room, const u32* off, const u32 children, const u32 segment, const u32 most, const u32 first_slot, const u32 first_child,
                                             const bool only, uint4* __restrict__ batches, Build_Counts* __restrict__ counts, u32* __restrict__ over, u32* __restrict__ left)
{
    const u32 tid = threadIdx.x;
    if(tid < (1 << MAX_B2) / 32) room.heads[tid] = 0;
    if(tid == 0) room.used = 0;
    for(u32 i = tid; i < children; i += blockDim.x) room.next[i] = u16(batch_end(off, i, children, segment, most));
    __syncthreads();
    for(u32 s = tid; s * segment < children; s += blockDim.x)
        for(u32 i = s * segment, end = min(children, (s + 1) * segment); i < end; i = room.next[i]) atomicOr(&room.heads[i >> 5], 1u << (i & 31u));
    __syncthreads();
    u32 mine = 0;       // up to two children a thread: whether a batch begins there
    #pragma unroll
    for(int h = 0; h < 2; ++h)
    {
        const u32 i = tid + h * blockDim.x;
        if(i >= children || !(room.heads[i >> 5] >> (i & 31u) & 1u)) continue;
        const u32 m = off[room.next[i]] - off[i];
        if(m > SORT_MOST)
        {
            if(m <= MEDIUM_CAP) left[atomicAdd(&counts->medium, 1u)] = children_entry(first_child + i, 1);
            else
            {
                over[atomicAdd(&counts->oversize, 1u)] = first_child + i;
                atomicAdd(&counts->oversize_records, m);
            }
        }
        else if(m) mine |= 1u << h;
    }
    u32 at = mine ? atomicAdd(&room.used, u32(__popc(mine))) : 0u;
    __syncthreads();
    if(tid == 0)
    {
        if(only) { room.at = 0; counts->batches = room.used; } else room.at = atomicAdd(&counts->batches, room.used);
    }
    __syncthreads();
    at += room.at;
    #pragma unroll
    for(int h = 0; h < 2; ++h)
        if(mine >> h & 1u)
        {
            const u32 i = tid + h * blockDim.x, e = room.next[i];
            batches[at++] = make_uint4(first_slot + off[i], off[e] - off[i], children_entry(first_child + i, e - i), 0);
        }
}

// Offsets of the parents and the work lists that follow from their sizes. one_level: there is no second split, the bins are
// the children of one parent that holds everything.
__global__ void __launch_bounds__(1024) parent_offsets_kernel(const u32* __restrict__ counts, const u32 bins, const u32 n, const int one_level, u32* __restrict__ cursor,
                                                             u32* __restrict__ par_off, u32* __restrict__ tile0, u32* __restrict__ child_off,
                                                             uint4* __restrict__ batches, u32* __restrict__ over, u32* __restrict__ left, const u32 split_tile, const u32 p, Build_Counts* __restrict__ stats)
{
    let_next_in();
    wait_for_previous();
    __shared__ u32 warp_tot[32];
    __shared__ u32 part[CSA_MAX_PARTITIONS];
    const u32 t = threadIdx.x;
    for(u32 i = t; i < p; i += 1024) part[i] = 0;
    const u32 c = t < bins ? (bins == 1 ? n : counts[t]) : 0;
    u32 total;
    const u32 off = block_exclusive<1024>(c, warp_tot, total);
    if(t < bins) cursor[t] = off;
    // the statistics' partitions: a bucket belongs to the p-th part of the suffix array in which it starts
    if(c) atomicAdd(&part[u64(off) * p / n], c);
    __syncthreads();
    u32 formed = 0, longest = 0;
    for(u32 i = t; i < p; i += 1024) { formed += part[i] != 0; longest = max(longest, part[i]); }
    if(formed) { atomicAdd(&stats->partitions, formed); atomicMax(&stats->max_partition, longest); }
    if(one_level)
    {
        __shared__ Batch_Room room;
        __shared__ u32 s_off[(1 << MAX_B1) + 1];
        if(t < bins) { child_off[t] = off; s_off[t] = off; }
        if(t == 0) { child_off[bins] = n; s_off[bins] = n; }
        __syncthreads();
        form_batches(room, s_off, bins, SHORT_SEGMENT, SHORT_BATCH, 0, 0, true, batches, stats, over, left);
        return;
    }
    const u32 tiles = (c + split_tile - 1) / split_tile;
    u32 all_tiles;
    const u32 t0 = block_exclusive<1024>(tiles, warp_tot, all_tiles);
    if(t < bins) { par_off[t] = off; tile0[t] = t0; }
    if(t == 0) { par_off[bins] = n; tile0[bins] = all_tiles; }
}

template <int BLOCK> constexpr size_t SCATTER_TEXT_SMEM = size_t(TILE_POSITIONS<BLOCK>) * 8;
static_assert(SCATTER_TEXT_SMEM<512> >= sizeof(Tile_Code<512>) && SCATTER_TEXT_SMEM<128> >= sizeof(Tile_Code<128>), "the windows lie where the records are staged later");

// Scatter by the top `bits` bits: the places inside a bucket come from shared-memory atomics and, for the tile's run of a bucket,
// from one global atomic (the order inside a bucket is free); records are staged in bucket order and written as runs. The global atomics are on their way from the moment that the counts
// are known, and waited for only behind the staging (with each waited for where it was made, as many after one another as a thread has buckets, 1.25e8 symbols took 0.52 ms instead of 0.51, and the split
// of the buckets 0.54 instead of 0.45). What bounds it is shared memory and L1 (80 % of their wavefronts): so a staged record carries its bin and its place in the tile in one word instead of its position and a bin beside it.
// keep_top: the record keeps the top bits (there is no second split), else its key starts behind them. PART: only the suffixes of the
// buckets [first_bin, first_bin + part_bins) are taken, and the cursors are theirs.
template <int BLOCK, bool PART>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) scatter_text_kernel(const u16* __restrict__ T, const u64 n, const u32* __restrict__ code, const int bits,
                                                                          const int keep_top, const u32 first_bin, const u32 part_bins, u32* __restrict__ cursor,
                                                                          u64* __restrict__ out)
{
    let_next_in();
    wait_for_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u64* const stage = reinterpret_cast<u64*>(smem_raw);
    static_assert(TILE_POSITIONS<BLOCK> <= 1 << 13 && MAX_B1 + 13 <= 32, "a staged record's lower word: its bin and its place in the tile");
    __shared__ u32 cnt[1 << MAX_B1];            // counts, then the bins' starts inside the tile
    __shared__ u32 base[1 << MAX_B1];           // where the tile's run of a bin goes, minus the run's start
    __shared__ u32 warp_tot[BLOCK / 32];
    const u32 bins = PART ? part_bins : 1u << bits;
    for(u32 i = threadIdx.x; i < bins; i += BLOCK) cnt[i] = 0;
    const u64 first = u64(blockIdx.x) * TILE_POSITIONS<BLOCK>;
    u32 ent[TEXT_ITEMS];
    u64 window = encode_tile<BLOCK>(T, n, first, code, *reinterpret_cast<Tile_Code<BLOCK>*>(smem_raw), ent);
    const u32 local = threadIdx.x * TEXT_ITEMS;
    const u64 room = n - first;
    const u32 valid = room < u64(TILE_POSITIONS<BLOCK>) ? u32(room) : u32(TILE_POSITIONS<BLOCK>);
    u32 key[TEXT_ITEMS], place[TEXT_ITEMS];      // place: bin << 16 | rank inside the tile's run of the bin
    u32 taken = 0;                               // a bit per suffix
    #pragma unroll
    for(int i = TEXT_ITEMS - 1; i >= 0; --i)
    {
        window = before(ent[i], window);
        const u32 high = u32(window >> 32), low = u32(window);
        const u32 bin = (bits ? high >> (32 - bits) : 0u) - (PART ? first_bin : 0u);
        key[i] = keep_top ? high : __funnelshift_l(low, high, bits);
        place[i] = bin << 16;
        if(local + i < valid && (!PART || bin < bins)) { place[i] |= atomicAdd(&cnt[bin], 1u); taken |= PART ? 1u << i : 0u; }
    }
    __syncthreads();
    constexpr int PER = (1 << MAX_B1) / BLOCK;      // bins per thread
    u32 mine[PER], got[PER], sum = 0;
    #pragma unroll
    for(int k = 0; k < PER; ++k) { const u32 b = threadIdx.x * PER + k; mine[k] = b < bins ? cnt[b] : 0; sum += mine[k]; }
    #pragma unroll
    for(int k = 0; k < PER; ++k) { got[k] = 0; if(mine[k]) got[k] = atomicAdd(&cursor[threadIdx.x * PER + k], mine[k]); }     // all on their way at once, and needed last
    u32 total;
    const u32 before_mine = block_exclusive<BLOCK>(sum, warp_tot, total);
    u32 run = before_mine;
    #pragma unroll
    for(int k = 0; k < PER; ++k)
    {
        const u32 b = threadIdx.x * PER + k;
        if(b < bins) cnt[b] = run;
        run += mine[k];
    }
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < TEXT_ITEMS; ++i)
        if(PART ? (taken >> i & 1u) != 0 : local + i < valid)
        {
            const u32 bin = place[i] >> 16;
            stage[cnt[bin] + (place[i] & 0xFFFFu)] = (u64(key[i]) << 32) | bin << 13 | (local + i);
        }
    run = before_mine;
    #pragma unroll
    for(int k = 0; k < PER; ++k)
    {
        const u32 b = threadIdx.x * PER + k;
        if(b < bins) base[b] = got[k] - run;
        run += mine[k];
    }
    __syncthreads();
    const u32 staged = PART ? total : valid;
    #pragma unroll 4
    for(u32 j = threadIdx.x; j < staged; j += BLOCK)
    {
        const u64 v = stage[j];
        out[base[u32(v) >> 13] + j] = (v & ~u64(0xFFFFFFFFu)) | u32(first + (u32(v) & 8191u));
    }
}

// ---- second split: every parent by the next bits ----------------------------------------------------------------------------------

// The parent whose run of blocks holds block `b` (first[p] <= b < first[p + 1]), found by all threads together; `found` is a
// word of shared memory. Returns parents if there is none. Ends with a barrier.
__device__ __forceinline__ u32 parent_of_block(const u32* __restrict__ first, const u32 parents, const u32 b, u32* found)
{
    if(threadIdx.x == 0) *found = parents;
    __syncthreads();
    for(u32 p = threadIdx.x; p < parents; p += blockDim.x)
        if(__ldg(first + p) <= b && b < __ldg(first + p + 1)) *found = p;
    __syncthreads();
    return *found;
}

template <int SPLIT_BLOCK>
__global__ void __launch_bounds__(SPLIT_BLOCK) count_children_kernel(const u64* __restrict__ rec, const u32* __restrict__ par_off, const u32* __restrict__ tile0,
                                                                    const u32 parents, const int bits, u32* __restrict__ counts)
{
    constexpr int SPLIT_TILE = SPLIT_BLOCK * SPLIT_ITEMS;
    __shared__ u32 cnt[1 << MAX_B2];
    __shared__ u32 found;
    let_next_in();
    wait_for_previous();
    const u32 children = 1u << bits;
    for(u32 i = threadIdx.x; i < children; i += SPLIT_BLOCK) cnt[i] = 0;
    const u32 p = parent_of_block(tile0, parents, blockIdx.x, &found);
    if(p >= parents) return;
    const u32 end = par_off[p + 1], first = par_off[p] + (blockIdx.x - tile0[p]) * SPLIT_TILE;
    const u32 valid = end - first < u32(SPLIT_TILE) ? end - first : u32(SPLIT_TILE);
    const u32* const words = reinterpret_cast<const u32*>(rec + first);
    u32 k[SPLIT_ITEMS];
    #pragma unroll
    for(int i = 0; i < SPLIT_ITEMS; ++i)
    {
        const u32 j = threadIdx.x + i * SPLIT_BLOCK;
        if(j < valid) k[i] = words[2 * j + 1];
    }
    #pragma unroll
    for(int i = 0; i < SPLIT_ITEMS; ++i)
        if(threadIdx.x + i * SPLIT_BLOCK < valid) atomicAdd(&cnt[k[i] >> (32 - bits)], 1u);
    __syncthreads();
    for(u32 i = threadIdx.x; i < children; i += SPLIT_BLOCK)
        if(cnt[i]) atomicAdd(&counts[u64(p) * children + i], cnt[i]);
}

// One block per parent: the children's counts become their places (in counts, running) and their offsets (child_off), and batches of the local sort.
__global__ void __launch_bounds__(1024) child_offsets_kernel(u32* __restrict__ counts, const u32* __restrict__ par_off, const u32 parents, const u32 children,
                                                            u32* __restrict__ child_off, uint4* __restrict__ batches, u32* __restrict__ over, u32* __restrict__ left, Build_Counts* __restrict__ stats)
{
    __shared__ u32 warp_tot[32];
    __shared__ u32 s_off[(1 << MAX_B2) + 1];
    __shared__ Batch_Room room;
    let_next_in();
    wait_for_previous();
    const u32 p = blockIdx.x, t = threadIdx.x;
    u32* const c = counts + u64(p) * children;
    const u32 i0 = 2 * t, i1 = 2 * t + 1;          // up to 2048 children
    const u32 a = i0 < children ? c[i0] : 0, b = i1 < children ? c[i1] : 0;
    u32 total;
    const u32 rel = block_exclusive<1024>(a + b, warp_tot, total), off = par_off[p] + rel;
    if(i0 < children) { c[i0] = off; child_off[u64(p) * children + i0] = off; s_off[i0] = rel; }
    if(i1 < children) { c[i1] = off + a; child_off[u64(p) * children + i1] = off + a; s_off[i1] = rel + a; }
    if(t == 0) s_off[children] = total;
    if(p == parents - 1 && t == 0) child_off[u64(parents) * children] = par_off[parents];
    __syncthreads();
    form_batches(room, s_off, children, SEGMENT, SORT_MOST, par_off[p], p * children, false, batches, stats, over, left);
}

template <int SPLIT_BLOCK> constexpr size_t SPLIT_SMEM = size_t(SPLIT_BLOCK * SPLIT_ITEMS) * 8;

template <int SPLIT_BLOCK>
__global__ void __launch_bounds__(SPLIT_BLOCK, 1024 / SPLIT_BLOCK) scatter_children_kernel(const u64* __restrict__ rec, const u32* __restrict__ par_off, const u32* __restrict__ tile0,
                                                                         const u32 parents, const int bits, u32* __restrict__ cursor, u64* __restrict__ out)
{
    constexpr int SPLIT_TILE = SPLIT_BLOCK * SPLIT_ITEMS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u64* const stage = reinterpret_cast<u64*>(smem_raw);
    __shared__ u32 cnt[1 << MAX_B2];
    __shared__ u32 base[1 << MAX_B2];
    __shared__ u32 warp_tot[SPLIT_BLOCK / 32];
    __shared__ u32 found;
    let_next_in();
    wait_for_previous();
    const u32 children = 1u << bits;
    for(u32 i = threadIdx.x; i < children; i += SPLIT_BLOCK) cnt[i] = 0;
    const u32 p = parent_of_block(tile0, parents, blockIdx.x, &found);
    if(p >= parents) return;
    const u32 end = par_off[p + 1], first = par_off[p] + (blockIdx.x - tile0[p]) * SPLIT_TILE;
    const u32 valid = end - first < u32(SPLIT_TILE) ? end - first : u32(SPLIT_TILE);
    u64 r[SPLIT_ITEMS];
    u32 place2[SPLIT_ITEMS / 2];         // ranks below 2^16, two a register
    #pragma unroll
    for(int i = 0; i < SPLIT_ITEMS; ++i)
    {
        const u32 j = threadIdx.x + i * SPLIT_BLOCK;
        if(j < valid) r[i] = rec[first + j];
    }
    #pragma unroll
    for(int i = 0; i < SPLIT_ITEMS; ++i)
    {
        u32 at = 0;
        if(threadIdx.x + i * SPLIT_BLOCK < valid) at = atomicAdd(&cnt[u32(r[i] >> 32) >> (32 - bits)], 1u);
        if(i & 1) place2[i >> 1] |= at << 16; else place2[i >> 1] = at;
    }
    __syncthreads();
    constexpr int PER = (1 << MAX_B2) / SPLIT_BLOCK;
    u32 mine[PER], got[PER], sum = 0;
    #pragma unroll
    for(int k = 0; k < PER; ++k) { const u32 b = threadIdx.x * PER + k; mine[k] = b < children ? cnt[b] : 0; sum += mine[k]; }
    #pragma unroll
    for(int k = 0; k < PER; ++k) { got[k] = 0; if(mine[k]) got[k] = atomicAdd(&cursor[u64(p) * children + threadIdx.x * PER + k], mine[k]); }      // all on their way at once, and needed last
    u32 total;
    const u32 before_mine = block_exclusive<SPLIT_BLOCK>(sum, warp_tot, total);
    u32 run = before_mine;
    #pragma unroll
    for(int k = 0; k < PER; ++k)
    {
        const u32 b = threadIdx.x * PER + k;
        if(b < children) cnt[b] = run;
        run += mine[k];
    }
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < SPLIT_ITEMS; ++i)
        if(threadIdx.x + i * SPLIT_BLOCK < valid)
            stage[cnt[u32(r[i] >> 32) >> (32 - bits)] + ((place2[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu)] = r[i];
    run = before_mine;
    #pragma unroll
    for(int k = 0; k < PER; ++k)
    {
        const u32 b = threadIdx.x * PER + k;
        if(b < children) base[b] = got[k] - run;
        run += mine[k];
    }
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < SPLIT_ITEMS; ++i)
    {
        const u32 j = threadIdx.x + i * SPLIT_BLOCK;
        if(j < valid)
        {
            const u64 v = stage[j];
            out[base[u32(v >> 32) >> (32 - bits)] + j] = v;
        }
    }
}

// ---- local sort: runs of children in shared memory --------------------------------------------------------------------------------

constexpr u32 TIE_ROOM = 1024;              // tied records that a block keeps before it writes them to the list
constexpr u32 MOST_CROWDED = 64;            // crowded bins of a batch
// A word holds the counts of four bins, five bits each, and later where the word's records begin (12 bits) and, in the fields, where those of each bin do.
constexpr u32 BIN_BITS = 5, BIN_MASK = (1u << BIN_BITS) - 1, START_BIT = 4 * BIN_BITS;
constexpr u32 each_bin(const u32 v) { return v | v << BIN_BITS | v << 2 * BIN_BITS | v << 3 * BIN_BITS; }
constexpr u32 SUMS = each_bin(1) << BIN_BITS;               // times a word of counts: the sums of the counts before each, and of all
constexpr u32 SUMS_BEFORE = each_bin(BIN_MASK) & ~BIN_MASK, SUM_OF_ALL = BIN_MASK << START_BIT;
constexpr u32 WINDOW_BIN = 4;               // records of the largest bin that a thread's window orders
constexpr u32 TO_EIGHT = each_bin(8 - WINDOW_BIN - 1), EIGHT_UP = each_bin(24);     // a count above WINDOW_BIN, the first added, has bits of the second
constexpr u32 FULL_BIN = each_bin(16);      // bits of a count from 16 on
static_assert(SORT_CAP <= 1 << (32 - START_BIT), "a slot takes 12 bits");
template <bool PACKED> constexpr size_t SORT_SMEM = (3 * SORT_CAP + 40) * 4 + TIE_ROOM * 8 + (PACKED ? SORT_BLOCK / 32 * 640 : 0);

__device__ __forceinline__ void order(u32& a, u32& b) { const u32 t = min(a, b); b = max(a, b); a = t; }
__device__ __forceinline__ void order(u32& a, u32& b, u32& c) { order(a, b); order(b, c); order(a, b); }

// A warp's entries [4 q0, 4 q0 + 128) of a batch go out, four a lane: the wanted ones of v. whole: the slot of the array that the batch's slot 0 is. words: 160 of the warp's in shared memory.
template <bool PACKED>
__device__ __forceinline__ void write_four(u32* const words, const u32 whole, const u32 q0, const u32 wanted, const uint4& v, u32* __restrict__ sa, u8* __restrict__ sa40)
{
    const u32 lane = lane_id(), first = whole + 4 * (q0 + lane);
    const u32 e[4] = {v.x, v.y, v.z, v.w};
    if(!PACKED)
    {
        if(wanted == 15u) *reinterpret_cast<uint4*>(sa + first) = v;
        else
            #pragma unroll
            for(u32 i = 0; i < 4; ++i)
                if(wanted >> i & 1u) sa[first + i] = e[i];
        return;
    }
    // four entries are 20 bytes, and begin on a word: the words of the warp's go out side by side
    u32* const w = words + 5 * lane;
    w[0] = v.x; w[1] = v.y << 8; w[2] = v.y >> 24 | v.z << 16; w[3] = v.z >> 16 | v.w << 24; w[4] = v.w >> 8;
    const u32 all_four = __ballot_sync(0xFFFFFFFFu, wanted == 15u);
    __syncwarp();
    u32* const to = reinterpret_cast<u32*>(sa40) + u64(whole / 4 + q0) * 5;
    #pragma unroll
    for(u32 j = lane; j < 160; j += 32)
        if(all_four >> (j / 5) & 1u) to[j] = words[j];
    if(wanted != 15u)
        #pragma unroll
        for(u32 i = 0; i < 4; ++i)
            if(wanted >> i & 1u)
            {
                u8* const b = sa40 + 5 * u64(first + i);
                b[0] = u8(e[i]); b[1] = u8(e[i] >> 8); b[2] = u8(e[i] >> 16); b[3] = u8(e[i] >> 24); b[4] = 0;
            }
    __syncwarp();
}

// ---- batches that lie unevenly ----------------------------------------------------------------------------------------------------------

constexpr u32 LEFT_BLOCKS = 148 * 2;        // of left_children_kernel, all resident
// Where large children are left for that kernel, batches are left beside them until it has so many. By 0, 148 and 296, a text of 4e6 tokens, uneven but independent: 508, 498 and 486 us, one in ten from the successors
// 528, 521 and 530, three in ten 570, 563 and 576; 2.2e6 and one in ten 440, 437 and 451. Where none are left, a chain of that kernel's would be added: 4e6 Zipf tokens 206 us, with batches left 213.
constexpr u32 LEFT_BESIDE = 148;
constexpr u32 SORT_RESIDENT = 148 * SORT_BLOCKS, SORT_GRID = SORT_RESIDENT * 8;         // blocks of the local sort at a time, and at most
constexpr u32 MOST_ROUNDS = (1u << (MAX_B1 + MAX_B2)) / SORT_GRID + 1, UNEVEN_WORDS = (MOST_ROUNDS + 8) / 32 + 2;          // batches of a block, and words of a bit for each and some behind them
constexpr u32 SORT_POS = 4 + SORT_CAP + 20, SORT_BINS = SORT_POS + SORT_CAP + 16;       // words of shared memory before the positions, before the bins
constexpr u32 STRETCH_BITS = 10;            // 1024 stretches: by 256, half as many crowded records again
constexpr u32 MOST_COMPARED = 48;           // comparisons a record, on average; by 16, 8e6 tokens of which six in ten come from successors take 965 us instead of 880 (the kernel behind does the rest)
// Of 256 records, those with the key of another beside them: from so many on the batch is left for its copies, and from fewer on if it cannot be done here. Builds of near-duplicates, by 16, 24 and 40: 2.9e6 tokens
// 1027, 1045 and 1043 us, 5.8e6 1097, 1104 and 1117; of dependent tokens (six in ten, 8e6) 851, 814 and 808.
constexpr u32 MANY_TWINS = 20, SOME_TWINS = 16;

// Keys of one batch from the start of the batch's range, which is cut to a power of two.
struct Batch_Keys
{
    u32 low; int up;
    __device__ __forceinline__ Batch_Keys(const u32 entry, const int bits)
    {
        const u32 others = entry & ((1u << MAX_B2) - 1);
        low = bits ? (entry >> MAX_B2 & ((1u << bits) - 1)) << (32 - bits) : 0u;
        up = bits - (32 - __clz(others));
    }
    __device__ __forceinline__ u32 operator()(const u32 key) const { return ((key - low) << up) & ~((1u << FREE_BITS) - 1); }
};

// A batch or a child goes to one of the kernels behind the local sort, by one thread; copies: many of its records have the same key, which is the second one's work.
__device__ __forceinline__ void leave_batch(const u32 children, const bool copies, Build_Counts* __restrict__ counts, u32* __restrict__ over, const u32 over_cap, u32* __restrict__ left)
{
    if(copies) over[over_cap - 1 - atomicAdd(&counts->crowded, 1u)] = children;
    else left[atomicAdd(&counts->medium, 1u)] = children;
}

// A batch whose keys lie unevenly in its range, as those of texts do whose symbols depend on the ones before. Its records are counted in 1024 stretches of the range first, and a stretch gets two bins a
// record. A record of a bin of up to WINDOW_BIN is compared with the others of its bin where it is; those of larger bins stand in a list, so that the threads of a warp have bins of one size as a rule.
// The array's entries are put together in shared memory, the tied records go to the list of the build at once. false: a bin of more than SMALL_GROUP records, or too many comparisons.
// What bounds it is the chain of ten steps between barriers, some 45,000 cycles for 2900 records where three blocks share an SM. Texts of 8e6 and 1.25e8 tokens, three in ten of which come from 32 successors of
// the one before: 685 us and 5.3 ms a build; every record compared with all of its bin by even bins (which the kernel behind does) 800 us and 6.2 ms, by that way alone 720 us and 5.8 ms. Crowded bins
// by a warp each, 16 steps a bin: 25,000 cycles of 75,000. Stretches with their least and largest key: a third fewer crowded records, but two more atomics for each.
template <bool PACKED>
__device__ __noinline__ bool spread_batch(const u64* __restrict__ rec, const u32 base, const u32 m, const u32 entry, const int bits, u32* __restrict__ sa, u8* __restrict__ sa40,
                                          u64* __restrict__ list, Build_Counts* __restrict__ counts)
{
    constexpr u32 BLOCK = SORT_BLOCK, ITEMS = SORT_ITEMS, CAP = SORT_CAP, WARPS = BLOCK / 32, PER = CAP / BLOCK;
    static_assert((1u << STRETCH_BITS) == 4 * BLOCK && 2 * CAP <= 1u << 13 && CAP <= 1u << 12 && PER % 4 == 0, "a thread sums four stretches; bins take 13 bits and slots 12");
    static_assert(CAP / (WINDOW_BIN + 1) <= 2 * TIE_ROOM && WINDOW_BIN == 4 && SMALL_GROUP <= 256 && (1u << STRETCH_BITS) <= CAP, "the lists and tables have room; sizes have their bits");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u32* const keys = reinterpret_cast<u32*>(smem_raw) + 4;             // [CAP] in the order of the bins; then the positions in their order
    u32* const pos = reinterpret_cast<u32*>(smem_raw) + SORT_POS;       // [CAP] of crowded bins' records
    u32* const bin = reinterpret_cast<u32*>(smem_raw) + SORT_BINS;      // [CAP] two 16-bit counts a word, then the bins' starts; then of every crowded record its bin, then where it goes
    u16* const start = reinterpret_cast<u16*>(bin);
    u32* const crowded = bin + CAP;                                     // of a crowded bin its first slot, its size - 1 << 12 and the crowded records before it << 20
    u16* const tie = reinterpret_cast<u16*>(crowded);                   // [CAP] then, by place, of a tied record TIED and the number of its group's before it, of a group's first HEAD and where the group goes
    u32* const words = crowded + 2 * TIE_ROOM + (threadIdx.x >> 5) * 160;       // PACKED: a warp's entries
    u32* const stretch = pos;                                           // [1024] records, later those before << 16
    __shared__ u32 warp_tot[WARPS], crowded_tot[WARPS];
    __shared__ u32 s_crowds, s_crowded, s_work, s_left, s_tied, s_slot, s_wide;
    const u32 tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, full = __shfl_sync(0xFFFFFFFFu, m / BLOCK, 0), rest = m % BLOCK, shift = base & 3u, end = shift + m, whole = base - shift;
    const Batch_Keys batch_key(entry, bits);
    auto for_each = [&](auto&& f)
    {
        #pragma unroll
        for(u32 i = 0; i < ITEMS - 1; ++i)
        {
            if(i >= full) break;
            f(i, tid + i * BLOCK);
        }
        if(tid < rest) f(ITEMS - 1, tid + full * BLOCK);
    };
    u32 k[ITEMS], p[ITEMS], at[ITEMS];          // at: the record's bin, and its number there << 13
    for_each([&](const u32 i, const u32 j) { const u64 v = rec[base + j]; k[i] = batch_key(u32(v >> 32)); p[i] = u32(v); });
    reinterpret_cast<uint4*>(stretch)[tid] = make_uint4(0, 0, 0, 0);
    for(u32 i = tid; 4 * i < m; i += BLOCK) reinterpret_cast<uint4*>(bin)[i] = make_uint4(0, 0, 0, 0);
    if(tid == 0) { s_work = 0; s_left = 0; s_tied = 0; s_wide = 0; }
    __syncthreads();
    for_each([&](const u32 i, const u32) { atomicAdd(stretch + (k[i] >> (32 - STRETCH_BITS)), 1u); });
    __syncthreads();
    {
        const uint4 v = reinterpret_cast<const uint4*>(stretch)[tid];
        const u32 sum = v.x + v.y + v.z + v.w, inc = warp_inclusive(sum);
        if(lane == 31) warp_tot[warp] = inc;
        __syncthreads();
        const u32 x = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? warp_tot[lane] : 0u) + inc - sum, y = x + v.x, z = y + v.y, w = z + v.z;
        reinterpret_cast<uint4*>(stretch)[tid] = make_uint4(x << 16 | v.x, y << 16 | v.y, z << 16 | v.z, w << 16 | v.w);
    }
    __syncthreads();
    for_each([&](const u32 i, const u32)
    {
        const u32 v = stretch[k[i] >> (32 - STRETCH_BITS)], b = 2 * (v >> 16) + __umulhi(k[i] << STRETCH_BITS, 2 * (v & 0xFFFFu));
        const u32 old = atomicAdd(bin + (b >> 1), (b & 1) ? 0x10000u : 1u);
        at[i] = b | ((b & 1) ? old >> 16 : old & 0xFFFFu) << 13;
    });
    __syncthreads();
    {
        u32 sum = 0, crowd = 0, work = 0, largest = 0;          // records, and crowded bins << 16; their records
        auto see = [&](const u32 c)
        {
            sum += c;
            if(c <= WINDOW_BIN) return;
            sum += 1u << 16;
            crowd += c;
            work += c * c;
            largest = max(largest, c);
        };
        #pragma unroll 1
        for(u32 w = 0; w < PER && tid * PER + w < m; w += 4)
        {
            const uint4 v = *reinterpret_cast<const uint4*>(bin + tid * PER + w);       // no bins behind 2 m, and zeros up to a multiple of four words
            see(v.x & 0xFFFFu); see(v.x >> 16); see(v.y & 0xFFFFu); see(v.y >> 16); see(v.z & 0xFFFFu); see(v.z >> 16); see(v.w & 0xFFFFu); see(v.w >> 16);
        }
        const u32 inc = warp_inclusive(sum), inc_crowd = warp_inclusive(crowd);
        work = __reduce_add_sync(0xFFFFFFFFu, work);
        if(lane == 31) { warp_tot[warp] = inc; crowded_tot[warp] = inc_crowd; }
        if(lane == 0 && work) atomicAdd(&s_work, work);
        if(largest > SMALL_GROUP) s_left = 1;
        __syncthreads();
        if(s_left || s_work > MOST_COMPARED * m) return false;
        u32 run = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? warp_tot[lane] : 0u) + inc - sum;
        u32 before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? crowded_tot[lane] : 0u) + inc_crowd - crowd, o = run >> 16;
        run = shift + (run & 0xFFFFu);
        auto note = [&](const u32 c)
        {
            if(c > WINDOW_BIN)
            {
                crowded[o++] = run | (c - 1) << 12 | before << 20;
                before += c;
            }
            run += c;
        };
        auto starts = [&](const u32 c) { const u32 v = run | (run + (c & 0xFFFFu)) << 16; note(c & 0xFFFFu); note(c >> 16); return v; };
        #pragma unroll 1
        for(u32 w = 0; w < PER && tid * PER + w < m; w += 4)
        {
            uint4 v = *reinterpret_cast<const uint4*>(bin + tid * PER + w);
            v.x = starts(v.x); v.y = starts(v.y); v.z = starts(v.z); v.w = starts(v.w);
            *reinterpret_cast<uint4*>(bin + tid * PER + w) = v;
        }
        if(tid == BLOCK - 1)
        {
            s_crowds = o;
            s_crowded = before;
            if(m % 4 == 0) bin[m] = run;        // the end behind the last bin; else it is in the last words above
        }
    }
    __syncthreads();
    constexpr u32 CROWDED = 1u << 16;           // at, from here on: the record's slot, its number in the bin << 12, the bin's size - 1 << 14; or this
    for_each([&](const u32 i, const u32)
    {
        const u32 b = at[i] & 0x1FFFu, number = at[i] >> 13, first = start[b], size = start[b + 1] - first, slot = first + number;
        keys[slot] = k[i];
        at[i] = slot | number << 12 | (size - 1) << 14;
        if(size > WINDOW_BIN) { pos[slot] = p[i]; at[i] = CROWDED; }
    });
    __syncthreads();
    #pragma unroll 1
    for(u32 o = tid; o < s_crowds; o += BLOCK)
    {
        const u32 size = (crowded[o] >> 12 & 255u) + 1, before = crowded[o] >> 20;
        #pragma unroll 4
        for(u32 i = 0; i < size; ++i) bin[before + i] = o;
    }
    u32 tied = 0;               // of the groups whose first record the thread has
    for_each([&](const u32 i, const u32)
    {
        const u32 slot = at[i] & 0xFFFu, number = at[i] >> 12 & 3u, last = at[i] >> 14;
        if(last == 0 || at[i] == CROWDED) { if(last == 0) at[i] = slot; return; }
        u32 less = 0, before = 0, group = 1;
        #pragma unroll
        for(u32 j = 0; j < WINDOW_BIN; ++j)
        {
            if(j > last) break;
            const u32 other = keys[slot - number + j];
            less += other < k[i];
            if(j != number && other == k[i]) { ++group; before += j < number; }
        }
        at[i] = (slot - number + less + before) | before << 12 | (group - 1) << 14;        // its place, the same before it, how many others are tied with it
        if(group > 1 && before == 0) tied += group;
    });
    __syncthreads();
    const u32 count = s_crowded;
    #pragma unroll 1
    for(u32 t = tid; t < count; t += BLOCK)
    {
        const u32 e = crowded[bin[t]], first = e & 0xFFFu, stop = first + (e >> 12 & 255u) + 1, slot = first + t - (e >> 20), key = keys[slot];
        u32 less = 0, upto = 0, before = 0;
        #pragma unroll 4
        for(u32 j = first; j < stop; ++j)
        {
            const u32 other = keys[j];
            if(j == slot) before = upto - less;
            less += other < key;
            upto += other <= key;
        }
        const u32 group = upto - less, place = first + less + before;
        // its place, its slot from there on << 12, and of a tied one the number of its group's before it or, of the first, behind it << 21
        bin[t] = place | (slot + 256 - place) << 12 | (group == 1 ? 0u : before ? before << 21 | 1u << 29 : (group - 1) << 21 | 3u << 29);
        if(group > 1 && before == 0)
        {
            tied += group;
            if(group > NARROW_GROUP) s_wide = 1;
        }
    }
    const u32 inc = warp_inclusive(tied);
    u32 to = 0;
    if(lane == 31 && inc) to = atomicAdd(&s_tied, inc);
    to = __shfl_sync(0xFFFFFFFFu, to, 31) + inc - tied;
    __syncthreads();
    u32 got = 0;                // on its way while the places are written
    if(tid == 0 && s_tied)
    {
        got = atomicAdd(&counts->small, s_tied);
        if(s_wide) counts->wide = 1;
    }
    constexpr u32 TIED = 1u << 15, HEAD = 1u << 14;
    for_each([&](const u32 i, const u32)
    {
        if(at[i] == CROWDED) return;
        const u32 place = at[i] & 0xFFFu, before = at[i] >> 12 & 3u, others = at[i] >> 14;
        keys[place] = p[i];
        tie[place] = u16(others == 0 ? 0u : before ? TIED | before : TIED | HEAD | to);
        if(others && before == 0) to += others + 1;
    });
    #pragma unroll 1
    for(u32 t = tid; t < count; t += BLOCK)
    {
        const u32 x = bin[t], place = x & 0xFFFu, number = x >> 21 & 255u;
        keys[place] = pos[place + (x >> 12 & 511u) - 256];
        tie[place] = u16((x >> 29 & 1u) == 0 ? 0u : (x >> 30) == 0 ? TIED | number : TIED | HEAD | to);
        if(x >> 30) to += number + 1;
    }
    if(tid == 0) s_slot = got;
    __syncthreads();
    u64* const ties = s_tied ? list + s_slot : nullptr;
    #pragma unroll 1
    for(u32 q0 = warp * 32; 4 * q0 < end; q0 += BLOCK)
    {
        const u32 q = q0 + lane;
        const uint4 x = reinterpret_cast<const uint4*>(keys)[q];
        u32 wanted = 4 * q < end ? 15u : 0u;
        if(4 * q < shift) wanted = 15u << shift & 15u;
        if(4 * q + 4 > end && wanted) wanted &= 15u >> (4 * q + 4 - end);
        u32 v[4] = {x.x, x.y, x.z, x.w};
        if(ties)
        {
            const uint2 w = reinterpret_cast<const uint2*>(tie)[q];
            const u32 e[4] = {w.x & 0xFFFFu, w.x >> 16, w.y & 0xFFFFu, w.y >> 16};
            #pragma unroll
            for(u32 i = 0; i < 4; ++i)
                if((wanted >> i & 1u) && (e[i] & TIED))
                {
                    const u32 before = e[i] & HEAD ? 0u : e[i] & 255u, head = 4 * q + i - before;
                    ties[(before ? tie[head] & (HEAD - 1) : e[i] & (HEAD - 1)) + before] = u64(whole + head) << 32 | v[i];
                    v[i] = SA_OPEN;
                }
        }
        write_four<PACKED>(words, whole, q0, wanted, make_uint4(v[0], v[1], v[2], v[3]), sa, sa40);
    }
    return true;
}

// The batches of a block that lie unevenly (a bit each in `uneven`). One of many batches goes to left_children_kernel, which does those of all blocks side by side: a block that has one when the others
// have ended takes another 15 us (1.25e8 tokens 2289 us a build, this way 2270). So do those of texts of one split (over_cap 0), which are few and small: that kernel has their largest children to do in
// any case, and does them beside those (1e5 tokens, three in ten from the successors, 158 us a build as here and 144 this way; 4e5 346 and 338, 2e6 484 and 492). Batches with many records of each key
// are another kernel's; where one after the other is, only one in eight is looked at.
template <bool PACKED>
__device__ __noinline__ void order_uneven(const u32* const uneven, const u64* __restrict__ rec, const uint4* __restrict__ batches, const u32 works, const int bits, u32* __restrict__ sa,
                                          u8* __restrict__ sa40, u64* __restrict__ list, Build_Counts* __restrict__ counts, u32* __restrict__ over, const u32 over_cap, u32* __restrict__ left)
{
    const u32 tid = threadIdx.x, rounds = (works - 1 - blockIdx.x) / gridDim.x + 1;
    auto lies_unevenly = [&](const u32 r) { return (uneven[r / 32] >> (r % 32) & 1u) != 0; };
    u32 all = 0;
    for(u32 w = 0; w < (rounds + 31) / 32; ++w) all += __popc(uneven[w]);
    if(8 * all < rounds || over_cap == 0)
    {
        for(u32 r = tid; r < rounds; r += SORT_BLOCK)
            if(lies_unevenly(r)) leave_batch(__ldg(&batches[blockIdx.x + r * gridDim.x].z), false, counts, over, over_cap, left);
        return;
    }
    u32 copied = 0;             // batches in a row that were left for their many records of each key
    #pragma unroll 1
    for(u32 r = 0; r < rounds; ++r)
    {
        if(!lies_unevenly(r)) continue;
        if(copied >= 2)
        {
            if(tid < 7 && r + tid < rounds && lies_unevenly(r + tid)) leave_batch(__ldg(&batches[blockIdx.x + (r + tid) * gridDim.x].z), true, counts, over, over_cap, left);
            r += 6;
            copied = 1;
            continue;
        }
        const uint4 batch = __ldg(batches + blockIdx.x + r * gridDim.x);
        // many records of each key, or keys that lie unevenly: how many of 32 records, eight times, have the key of another?
        if(16 * tid < batch.y) asm volatile("prefetch.global.L2 [%0];" :: "l"(rec + batch.x + 16 * tid));
        const bool looked_at = tid < batch.y;
        const u64 key = looked_at ? rec[batch.x + tid] >> 32 : ~u64(tid);
        const u32 alike = __popc(__match_any_sync(0xFFFFFFFFu, key));
        const u32 twins = __syncthreads_count(looked_at && alike > 1);
        const bool copies = twins >= MANY_TWINS;
        copied = copies ? copied + 1 : 0;
        // the first few go beside what the kernel behind has to do in any case
        const bool room = __syncthreads_or(tid == 0 && !copies && __ldcg(&counts->medium) - 1 < LEFT_BESIDE - 1);
        const bool done = !copies && !room && spread_batch<PACKED>(rec, batch.x, batch.y, batch.z, bits, sa, sa40, list, counts);
        if(tid == 0 && !done) leave_batch(batch.z, twins >= SOME_TWINS, counts, over, over_cap, left);
    }
}

// ---- the local sort ------------------------------------------------------------------------------------------------------------------------

// A batch goes through four steps with a barrier behind each:
//   * every record is counted in a bin, its key's place in the batch's range of keys by interpolation (two bins to a record), and keeps its number in the bin;
//   * the bins' counts become their starts;
//   * key and position go to the record's slot in shared memory. The keys are in order now but for bins with several records, most of which hold two to four;
//   * a thread orders the keys of four slots with those of the three slots before and behind, in registers: a bin of up to four records lies inside the window of every
//     slot of it. A key carries its slot's last four bits in bits that it does not need, so min and max move whole records, and no two are equal. The four entries go out
//     as one 16-byte store: the batch's slots begin with the first slot's place in its group of four.
// The one or two larger bins of a batch, of up to 15 records, are ordered by a warp each. Batches with a bin of 16 or more, with crowded bins all over or with too many tied records wait until the block has
// tried its others (order_uneven): the registers of a kernel that orders them where they turn up cost even texts 4 to 5 %.
// What bounds it: the issue of instructions (110 for 32 records, 59 % of the cycles) and the latency of dependent steps between barriers; so records stay in registers, no slow path is
// unrolled, a block's next records and the batch after them are on their way early, and 256 threads with 16 records each share what a warp does per batch among more records than 512
// with 8 do. A Zipf text of 1.25e8 symbols, the kernel alone: 0.66 ms; 512 threads with 8 records, two blocks an SM 0.78 and three (40 registers, spills) 1.0; two blocks of 256
// 0.74; all keys of a bin compared with one another and every record placed by its rank (226 instructions) 1.14. Room for 2048 tied records instead of 1024 leaves L1 too small for
// the registers that spill: 1 % of a build.
// PACKED: the array is written to sa40 as 5-byte entries, else to sa. over_cap: 0 where crowded_batches_kernel is not launched.
template <bool PACKED>
__global__ void __launch_bounds__(SORT_BLOCK, SORT_BLOCKS) local_sort_kernel(const u64* __restrict__ rec, const uint4* __restrict__ batches, const int bits, u32* __restrict__ sa,
                                                                             u8* __restrict__ sa40, u64* __restrict__ list, Build_Counts* __restrict__ counts, u32* __restrict__ over,
                                                                             const u32 over_cap, u32* __restrict__ left)
{
    constexpr u32 BLOCK = SORT_BLOCK, ITEMS = SORT_ITEMS, CAP = SORT_CAP, WARPS = BLOCK / 32, WORDS = CAP / 2 / BLOCK, CROWD_WORDS = CAP / 32 + 4;
    static_assert(WORDS % 4 == 0 && ITEMS % 8 == 0 && CROWD_WORDS <= BLOCK, "whole 16-byte pieces of bins, whole words of numbers, a word of marks a thread");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u32* const keys = reinterpret_cast<u32*>(smem_raw) + 4;     // [CAP + 16] in the order of the bins; four words before it
    u32* const pos = reinterpret_cast<u32*>(smem_raw) + SORT_POS;       // [CAP + 16] the positions beside them; four words before it
    u32* const bins = reinterpret_cast<u32*>(smem_raw) + SORT_BINS;     // [2][CAP / 2]: of every other batch
    u64* const tie = reinterpret_cast<u64*>(bins + CAP);        // [TIE_ROOM]
    u32* const words = reinterpret_cast<u32*>(tie + TIE_ROOM) + (threadIdx.x >> 5) * 160;       // PACKED: a warp's entries
    __shared__ u32 warp_tot[WARPS];
    __shared__ u32 crowd[CROWD_WORDS];              // a bit per slot: it belongs to a crowded bin
    __shared__ u32 crowded[MOST_CROWDED];           // such a bin's first slot and its size
    __shared__ u32 s_crowded, s_fall[2], s_ties, s_slot;
    __shared__ u32 s_uneven[UNEVEN_WORDS];          // a bit per batch of the block: it lies unevenly (bits behind its last may stand, too)
    __shared__ u32 s_some_uneven, s_round, s_next_round;    // which of the block's batches this one and the next are
    __shared__ u32 s_before;                        // the round of the batch before
    const u32 tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    let_next_in();
    wait_for_previous();
    const uint2 found = __ldcg(reinterpret_cast<const uint2*>(&counts->batches));
    const u32 works = found.x;
    if(blockIdx.x >= works) return;

    u32 k[ITEMS], p[ITEMS];
    u32 full = 0, rest = 0;             // rows of the batch that have a record for every thread, and records behind them
    auto for_each = [&](auto&& f)
    {
        #pragma unroll
        for(u32 i = 0; i < ITEMS - 1; ++i)
        {
            if(i >= full) break;
            f(i);
        }
        if(tid < rest) f(ITEMS - 1);
    };
    auto load = [&](const uint4& batch)
    {
        full = __shfl_sync(0xFFFFFFFFu, batch.y / BLOCK, 0);
        rest = batch.y % BLOCK;
        const u64* const at = rec + batch.x + tid;
        #pragma unroll
        for(u32 i = 0; i < ITEMS - 1; ++i)
        {
            if(i >= full) break;
            const u64 v = at[i * BLOCK];
            k[i] = u32(v >> 32); p[i] = u32(v);
        }
        if(tid < rest) { const u64 v = at[full * BLOCK]; k[ITEMS - 1] = u32(v >> 32); p[ITEMS - 1] = u32(v); }
    };
    auto put = [&](const u32 slot, const u32 v)
    {
        if(!PACKED) { sa[slot] = v; return; }
        u8* const b = sa40 + 5 * u64(slot);
        b[0] = u8(v); b[1] = u8(v >> 8); b[2] = u8(v >> 16); b[3] = u8(v >> 24); b[4] = 0;
    };

    uint4 now = __ldg(batches + blockIdx.x), then = make_uint4(0, 0, 0, 0);
    load(now);
    const u32 tries = tid == 0 && blockIdx.x % 8 ? found.y : 0u;
    for(u32 i = tid; i < CAP / 4; i += BLOCK) reinterpret_cast<uint4*>(bins)[i] = make_uint4(0, 0, 0, 0);
    if(tid < 4) keys[int(tid) - 4] = 0;
    if(tid < UNEVEN_WORDS) s_uneven[tid] = 0;
    if(tid == 0) { s_fall[0] = 0; s_ties = 0; s_round = 0; s_next_round = 1; s_some_uneven = 0; }
    u32 turn = 0, kept = 0;             // kept: tied records in `tie` from before the batch
    u32 next = blockIdx.x + gridDim.x, fell = 0;        // fell: batches in a row that are not done here
    // One block in eight tries its first batch in any case. Where most of those that have come to an end did not do it, the others do not try their first seven (1e7 tokens of which most stand five times: some 40 us of 1320).
    if(__syncthreads_or(2 * (tries & 0xFFFFu) > tries >> 16))
    {
        if(tid == 0) { s_uneven[0] = 127; s_some_uneven = 1; s_round = 7; s_next_round = 8; }
        next += 7 * gridDim.x; fell = 7;
        now.y = 0;
        if(next - gridDim.x < works) { now = __ldg(batches + (next - gridDim.x)); load(now); }
    }
    if(next < works) then = __ldg(batches + next);
    while(now.y)
    {
        const u32 base = now.x, m = now.y, shift = base & 3u, end = shift + m;      // the batch's records take the slots [shift, end)
        const u32 whole = base - shift;
        u32* const bin = bins + turn * (CAP / 2);
        {
            const Batch_Keys batch_key(now.z, bits);
            for_each([&](const u32 i) { k[i] = batch_key(k[i]); });
        }
        u32 seen = 0, number[ITEMS / 8] = {};       // the records' numbers in their bins, four bits each
        for_each([&](const u32 i)
        {
            const u32 b = __umulhi(k[i], 2 * m), old = atomicAdd(bin + (b >> 2), 1u << (BIN_BITS * (b & 3u)));
            seen |= old;
            number[i / 8] |= (old >> (BIN_BITS * (b & 3u)) & 15u) << (4 * (i % 8));
        });
        if(seen & FULL_BIN) s_fall[turn] = 1;       // before a count runs into the next
        __syncthreads();

        const bool any = 2 * WORDS * tid < m;       // the thread has bins, its warp has
        const bool busy = 64 * WORDS * warp < m;
        u32 c[WORDS], sum = 0, inc = 0, many = 0;
        if(busy)
        {
            #pragma unroll
            for(u32 w = 0; w < WORDS; w += 4)
            {
                const uint4 v = any ? *reinterpret_cast<const uint4*>(bin + WORDS * tid + w) : make_uint4(0, 0, 0, 0);
                c[w] = v.x; c[w + 1] = v.y; c[w + 2] = v.z; c[w + 3] = v.w;
            }
            #pragma unroll
            for(u32 w = 0; w < WORDS; ++w)
            {
                many |= (c[w] + TO_EIGHT) & EIGHT_UP;
                sum += c[w] * SUMS & SUM_OF_ALL;
            }
            inc = warp_inclusive(sum);
        }
        if(lane == 31) warp_tot[warp] = inc;
        // what the batch before has left: its marks, and its ties where the next might find no room for its own
        #pragma unroll
        for(u32 w = 0; w < WORDS; w += 4) reinterpret_cast<uint4*>(bins + (turn ^ 1) * (CAP / 2))[tid + w / 4 * BLOCK] = make_uint4(0, 0, 0, 0);
        if(tid < CROWD_WORDS) crowd[tid] = 0;
        const bool crammed = s_ties > TIE_ROOM;             // to be done again
        const u32 ties = crammed ? kept : s_ties;
        const bool write = ties != 0 && (crammed || ties + max(TIE_ROOM / 4, 2 * (ties - kept)) > TIE_ROOM);
        if(tid == 0)
        {
            s_crowded = 0;
            s_fall[turn ^ 1] = 0;
            if(crammed) { s_uneven[s_before >> 5] |= 1u << (s_before & 31u); s_some_uneven = 1; }
            s_before = s_round;
            if(write) s_slot = atomicAdd(&counts->small, ties);
        }
        __syncthreads();
        if(16 * tid < then.y) asm volatile("prefetch.global.L2 [%0];" :: "l"(rec + then.x + 16 * tid));
        if(busy)
        {
            u32 run = (shift << START_BIT) + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? warp_tot[lane] : 0u) + inc - sum;
            if(any)
            {
                #pragma unroll
                for(u32 w = 0; w < WORDS; w += 4)
                {
                    uint4 v;
                    v.x = (c[w] * SUMS & SUMS_BEFORE) | run; run += c[w] * SUMS & SUM_OF_ALL;
                    v.y = (c[w + 1] * SUMS & SUMS_BEFORE) | run; run += c[w + 1] * SUMS & SUM_OF_ALL;
                    v.z = (c[w + 2] * SUMS & SUMS_BEFORE) | run; run += c[w + 2] * SUMS & SUM_OF_ALL;
                    v.w = (c[w + 3] * SUMS & SUMS_BEFORE) | run; run += c[w + 3] * SUMS & SUM_OF_ALL;
                    *reinterpret_cast<uint4*>(bin + WORDS * tid + w) = v;
                }
            }
            if(many)
            {
                #pragma unroll
                for(u32 w = 0; w < WORDS; ++w)
                    #pragma unroll 1
                    for(u32 f = (c[w] + TO_EIGHT) & EIGHT_UP; f;)
                    {
                        const u32 bit = (__ffs(f) - 1) / BIN_BITS * BIN_BITS, size = c[w] >> bit & BIN_MASK, v = bin[WORDS * tid + w];
                        const u32 at = (v >> START_BIT) + (v >> bit & BIN_MASK), o = atomicAdd(&s_crowded, 1u);
                        f &= ~(BIN_MASK << bit);
                        if(o < MOST_CROWDED) crowded[o] = at | size << 16;
                        const u64 marks = u64((1u << size) - 1) << (at & 31u);
                        atomicOr(&crowd[at >> 5], u32(marks));
                        if(marks >> 32) atomicOr(&crowd[(at >> 5) + 1], u32(marks >> 32));
                        u32 all = 0;
                        for(int b = 0; b < 4; ++b) all += c[w] >> (BIN_BITS * b) & BIN_MASK;
                        if(o >= MOST_CROWDED || (c[w] & FULL_BIN) || all > BIN_MASK) s_fall[turn] = 1;
                    }
            }
        }
        if(write)
            #pragma unroll 1
            for(u32 j = tid; j < ties; j += BLOCK) list[u64(s_slot) + j] = tie[j];
        kept = write ? 0 : ties;
        __syncthreads();

        const bool fall = s_fall[turn] != 0;
        if(tid == 0 && (write || crammed)) s_ties = kept;
        if(!fall)
        {
            for_each([&](const u32 i)
            {
                const u32 b = __umulhi(k[i], 2 * m), v = bin[b >> 2], slot = (v >> START_BIT) + (v >> (BIN_BITS * (b & 3u)) & BIN_MASK) + (number[i / 8] >> (4 * (i % 8)) & 15u);
                keys[slot] = k[i] | (slot & 15u);
                pos[slot] = p[i];
            });
            if(tid < shift) keys[tid] = 0;                      // no key is below, or above those behind
            if(tid < 8) keys[end + tid] = 0xFFFFFFFFu;
        }
        else if(tid == 0) { s_uneven[s_round >> 5] |= 1u << (s_round & 31u); s_some_uneven = 1; }
        __syncthreads();

        if(next < works) load(then);            // on their way while the batch is ordered
        if(!fall)
        {
            const u32 crowds = s_crowded;
            #pragma unroll 1
            for(u32 q0 = warp * 32; 4 * q0 < end; q0 += BLOCK)
            {
                const u32 q = q0 + lane, window = 4 * q - 3;
                const uint4* const K = reinterpret_cast<const uint4*>(keys - 4) + q;
                const uint4 L = K[0], O = K[1], R = K[2];
                u32 a0 = L.y, a1 = L.z, a2 = L.w, x0 = O.x, x1 = O.y, x2 = O.z, x3 = O.w, r0 = R.x, r1 = R.y, r2 = R.z;
                order(x0, x1); order(x2, x3); order(x0, x2); order(x1, x3); order(x1, x2);
                order(a0, a1, a2);
                order(r0, r1, r2);
                const u32 before = max(max(min(a0, x2), min(a1, x1)), min(a2, x0));        // the key at the place before the four, and the one behind them
                x2 = max(a0, x2); x1 = max(a1, x1); x0 = max(a2, x0);
                order(x0, x1, x2);
                const u32 behind = min(min(max(x1, r2), max(x2, r1)), max(x3, r0));
                x1 = min(x1, r2); x2 = min(x2, r1); x3 = min(x3, r0);
                order(x1, x2, x3);
                const u32* const at = pos + 4 * q - 3;
                u32 v[4] = {at[(x0 - window) & 15u], at[(x1 - window) & 15u], at[(x2 - window) & 15u], at[(x3 - window) & 15u]};
                u32 wanted = 4 * q < end ? 15u : 0u;            // a bit per entry: it is the batch's, and of no crowded bin
                if(4 * q < shift) wanted = 15u << shift & 15u;
                if(4 * q + 4 > end && wanted) wanted &= 15u >> (4 * q + 4 - end);
                if(crowds) wanted &= ~(crowd[q >> 3] >> (4 * (q & 7u)));
                const u32 x[6] = {before, x0, x1, x2, x3, behind};
                bool tied = min(min(min(before ^ x0, x0 ^ x1), min(x1 ^ x2, x2 ^ x3)), x3 ^ behind) < 16;
                if(tied && wanted != 15u)       // the words around the batch are alike
                {
                    tied = false;
                    #pragma unroll
                    for(u32 i = 0; i < 4; ++i)
                        tied |= (wanted >> i & 1u) && (((x[i] ^ x[i + 1]) < 16 && 4 * q + i > shift) || ((x[i + 1] ^ x[i + 2]) < 16 && 4 * q + i + 1 < end));
                }
                if(tied)
                {
                    #pragma unroll
                    for(u32 i = 0; i < 4; ++i)
                    {
                        if(!(wanted >> i & 1u) || ((x[i] ^ x[i + 1]) >= 16 && (x[i + 1] ^ x[i + 2]) >= 16)) continue;
                        const u32 first = max(4 * q + i, shift + 3) - 3, stop = min(4 * q + i + 4, end);
                        u32 smaller = 0, group = 0;
                        #pragma unroll 1
                        for(u32 s = first; s < stop; ++s)
                            if((keys[s] ^ x[i + 1]) < 16) { ++group; smaller += keys[s] < x[i + 1]; }
                        if(group <= 1) continue;
                        v[i] = SA_OPEN;
                        if(smaller) continue;            // the first of a group writes it
                        u32 o = atomicAdd(&s_ties, group);
                        if(o + group > TIE_ROOM) continue;
                        #pragma unroll 1
                        for(u32 s = first; s < stop; ++s)
                            if((keys[s] ^ x[i + 1]) < 16) tie[o++] = u64(whole + 4 * q + i) << 32 | pos[s];
                    }
                }
                write_four<PACKED>(words, whole, q0, wanted, make_uint4(v[0], v[1], v[2], v[3]), sa, sa40);
            }
            #pragma unroll 1
            for(u32 o = WARPS - 1 - warp; o < crowds; o += WARPS)       // the last warps have the fewest windows
            {
                const u32 s = crowded[o] & 0xFFFFu, size = crowded[o] >> 16;
                const bool mine = lane < size;
                const u32 key = mine ? keys[s + lane] >> FREE_BITS : ~0u, at = mine ? pos[s + lane] : 0u;
                u32 less = 0, equal = 0;
                #pragma unroll 4
                for(u32 j = 0; j < 16; ++j)
                {
                    const u32 other = __shfl_sync(0xFFFFFFFFu, key, j);
                    less += other < key;
                    equal |= u32(other == key) << j;
                }
                const u32 before = __popc(equal & ((1u << lane) - 1u)), group = __popc(equal);
                u32 to = 0;
                if(mine && group > 1 && before == 0) to = atomicAdd(&s_ties, group);
                to = __shfl_sync(0xFFFFFFFFu, to, max(__ffs(equal), 1) - 1);
                if(mine)
                {
                    const u32 head = whole + s + less;
                    put(head + before, group > 1 ? SA_OPEN : at);
                    if(group > 1 && to + group <= TIE_ROOM) tie[to + before] = u64(head) << 32 | at;
                }
            }
        }
        if(next >= works) break;
        now = then;
        // where one batch after the other is not done here, only one in eight is tried
        fell = fall || crammed ? fell + 1 : 0;
        const u32 jump = fell < 2 ? 1u : 8u;
        if(tid == 0)
        {
            const u32 passed = s_next_round + 1;
            if(jump == 8) { s_uneven[passed >> 5] |= 127u << (passed & 31u); s_uneven[(passed >> 5) + 1] |= u32(127ull << (passed & 31u) >> 32); }
            s_round = s_next_round;
            s_next_round += jump;
        }
        next += jump * gridDim.x;
        then.y = 0;
        if(next < works) then = __ldg(batches + next);
        turn ^= 1;
    }
    __syncthreads();
    const bool crammed = s_ties > TIE_ROOM;
    const u32 ties = crammed ? kept : s_ties;
    if(tid == 0)
    {
        if(crammed) { s_uneven[s_round >> 5] |= 1u << (s_round & 31u); s_some_uneven = 1; }
        if(blockIdx.x % 8 == 0) atomicAdd(&counts->tries, 1u << 16 | (s_uneven[0] & 1u));
        if(ties) s_slot = atomicAdd(&counts->small, ties);
    }
    __syncthreads();
    #pragma unroll 1
    for(u32 j = tid; j < ties; j += BLOCK) list[u64(s_slot) + j] = tie[j];
    if(s_some_uneven) order_uneven<PACKED>(s_uneven, rec, batches, works, bits, sa, sa40, list, counts, over, over_cap, left);
}

// ---- crowded batches ------------------------------------------------------------------------------------------------------------------

constexpr u32 CROWD_BLOCK = 256, CROWD_ITEMS = 16, CROWD_CAP = CROWD_BLOCK * CROWD_ITEMS;
constexpr u32 MOST_KEYS = 16;               // a bin with more keys: the batch goes on to the kernel behind this one
constexpr size_t CROWD_SMEM = size_t(CROWD_CAP) * (4 + 2 * 5 + 4);
static_assert(CROWD_CAP > SORT_MOST && CROWD_CAP <= 4096, "a record's number in its batch takes 12 bits, with two flags and one pattern to spare in 16");

// Batches in which many records have the same key (near-duplicate documents: some fifty a key). A key is ordered once, however many records have it: each round, the records that have
// no key yet write themselves into their bin of the interpolation; the one that stands there then brings its key, and those of the same key are counted for it and numbered. One round does
// for all but a few records as a rule; those left over go on as a list. The keys of a bin, one a round, are a list too: a key's place is behind the smaller ones of its list and the bins before, and a
// record's is its key's and its number.
// Bound by the issue of instructions (178 for 32 records) and the latency of its steps: 0.54 ms for 6e7 near-duplicate suffixes where the kernel that compares all records of a bin takes 1.9 ms (the build of
// 4e8 of them 60.5 -> 52.6 ms).
template <bool PACKED>
__global__ void __launch_bounds__(CROWD_BLOCK, 3) crowded_batches_kernel(const u64* __restrict__ rec, const int bits, const u32* __restrict__ child_off, u32* __restrict__ sa, u8* __restrict__ sa40,
                                                                         u64* __restrict__ list, const u64 list_cap, Build_Counts* __restrict__ counts, const u32* __restrict__ over,
                                                                         const u32 over_cap, u32* __restrict__ left)
{
    constexpr u32 BLOCK = CROWD_BLOCK, ITEMS = CROWD_ITEMS, CAP = CROWD_CAP, WORDS = CAP / 2 / BLOCK, NONE = 0xFFFFu, SETTLED = 1u << 12, WON = 1u << 13, RECORD = SETTLED - 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u32* const keys = reinterpret_cast<u32*>(smem_raw);                 // [CAP] of the records; then positions of tied ones
    u32* const res = keys + CAP;                                        // [CAP] place of the key that the record brought; of a record of the list: its key's record and its number << 16, or
                                                                        // its key's place, its number << 16 and bit 31 where it brought the key
    u32* const bin = res + CAP;                                         // [CAP / 2] two 16-bit counts a word: records of each bin, then the bins' starts
    u16* const start = reinterpret_cast<u16*>(bin);                     // at first who stands in the bin
    u16* const head = start + CAP;                                      // [CAP] the last key of every bin's list, by its record
    u32* const heads = bin;                                             // [CAP] both, when they are done with: first slots of tied records
    u32* const cnt2 = bin + CAP;                                        // [CAP / 2] two 16-bit counts a word: records of each key
    u16* const cnt = reinterpret_cast<u16*>(cnt2);
    u16* const link = cnt + CAP;                                        // [CAP] the key before it in its list; then where its records go among the tied ones
    u16* const lines = link + CAP;                                      // [CAP] records without a key after the first round, from the front; those that brought one in it, from the back
    __shared__ u32 warp_tot[BLOCK / 32];
    __shared__ u32 s_lines, s_tied[2], s_slot[2];
    __shared__ u32 s_wide;      // told once a block: with a store a key to the one word, builds of near-duplicates wait for it
    const u32 tid = threadIdx.x, lane = lane_id();
    auto put = [&](const u32 slot, const u32 v)
    {
        if(!PACKED) { sa[slot] = v; return; }
        u8* const b = sa40 + 5 * u64(slot);
        b[0] = u8(v); b[1] = u8(v >> 8); b[2] = u8(v >> 16); b[3] = u8(v >> 24); b[4] = 0;
    };
    let_next_in();
    wait_for_previous();
    const u32 works = counts->crowded;
    if(blockIdx.x >= works) return;
    // the batch and the one after it, whose records are on their way while the one before is finished
    u32 entry = over[over_cap - 1 - blockIdx.x], next_entry = 0, next_base = 0, next_end = 0;
    u32 base = __ldg(child_off + (entry >> MAX_B2)), m = __ldg(child_off + (entry >> MAX_B2) + (entry & ((1u << MAX_B2) - 1)) + 1) - base;
    u32 k[ITEMS], p[ITEMS];
    auto load = [&]()
    {
        #pragma unroll
        for(u32 i = 0; i < ITEMS; ++i)
        {
            if(i * BLOCK >= m) break;
            const u32 j = tid + i * BLOCK;
            if(j < m) { const u64 v = rec[base + j]; k[i] = u32(v >> 32); p[i] = u32(v); }
        }
    };
    load();
    if(tid == 0) s_wide = 0;    // several barriers before it is told
    for(u32 work = blockIdx.x; work < works; work += gridDim.x)
    {
        const u32 others = entry & ((1u << MAX_B2) - 1), low = bits ? (entry >> MAX_B2 & ((1u << bits) - 1)) << (32 - bits) : 0u;
        const int up = bits - (32 - __clz(others));
        const bool more_work = work + gridDim.x < works;
        if(more_work) next_entry = over[over_cap - 1 - work - gridDim.x];
        auto for_each = [&](auto&& f)
        {
            #pragma unroll
            for(u32 i = 0; i < ITEMS; ++i)
            {
                if(i * BLOCK >= m) break;
                if(tid + i * BLOCK < m) f(i, tid + i * BLOCK);
            }
        };
        for(u32 i = tid; i < (m + 7) / 8; i += BLOCK)
        {
            reinterpret_cast<uint4*>(head)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
            reinterpret_cast<uint4*>(cnt2)[i] = make_uint4(0, 0, 0, 0);
        }
        if(tid == 0) s_lines = 0;
        if(tid < 2) s_tied[tid] = 0;
        u32 key_of[ITEMS];      // the record that brought the key, and the number << 16
        for_each([&](const u32 i, const u32 j)
        {
            k[i] = (k[i] - low) << up;
            keys[j] = k[i];
            start[__umulhi(k[i], m)] = u16(j);
        });
        __syncthreads();
        u32 won = 0, open = 0;
        for_each([&](const u32 i, const u32 j)
        {
            const u32 b = __umulhi(k[i], m), e = start[b];
            if(keys[e] == k[i])
            {
                const u32 number = atomicAdd(&cnt2[e >> 1], (e & 1) ? 0x10000u : 1u);
                key_of[i] = e | ((e & 1) ? number & 0xFFFF0000u : number << 16);
                if(e == j) { head[b] = u16(e); link[e] = u16(NONE); won |= 1u << i; }
            }
            else open |= 1u << i;
        });
        {
            const u32 mine = __popc(open) | __popc(won) << 16, inc = warp_inclusive(mine);
            u32 at = 0;
            if(lane == 31) at = atomicAdd(&s_lines, inc);
            at = __shfl_sync(0xFFFFFFFFu, at, 31) + inc - mine;
            u32 front = at & 0xFFFFu, back = CAP - 1 - (at >> 16);
            if(mine) for_each([&](const u32 i, const u32 j)
            {
                if(open >> i & 1u) lines[front++] = u16(j);
                else if(won >> i & 1u) lines[back--] = u16(j);
            });
        }
        __syncthreads();
        const u32 open_ones = s_lines & 0xFFFFu, winners = s_lines >> 16;
        u32 rounds = 1;
        for(bool more = open_ones != 0; more; ++rounds)
        {
            if(rounds == MOST_KEYS) break;
            #pragma unroll 1
            for(u32 t = tid; t < open_ones; t += BLOCK)
            {
                const u32 j = lines[t];
                if(!(j & SETTLED)) start[__umulhi(keys[j], m)] = u16(j);
            }
            __syncthreads();
            bool here = false;
            #pragma unroll 1
            for(u32 t = tid; t < open_ones; t += BLOCK)
            {
                const u32 j = lines[t];
                if(j & SETTLED) continue;
                const u32 key = keys[j], b = __umulhi(key, m), e = start[b];
                if(keys[e] != key) { here = true; continue; }
                const u32 number = atomicAdd(&cnt2[e >> 1], (e & 1) ? 0x10000u : 1u);
                res[j] = e | ((e & 1) ? number & 0xFFFF0000u : number << 16);
                if(e == j) { link[e] = head[b]; head[b] = u16(e); }
                lines[t] = u16(j | SETTLED | (e == j ? WON : 0u));
            }
            more = __syncthreads_or(here);
        }
        if(more_work)
        {
            next_base = __ldg(child_off + (next_entry >> MAX_B2));
            next_end = __ldg(child_off + (next_entry >> MAX_B2) + (next_entry & ((1u << MAX_B2) - 1)) + 1);
        }
        auto go_on = [&]() { entry = next_entry; base = next_base; m = next_end - next_base; if(more_work) load(); };
        if(rounds == MOST_KEYS)
        {
            if(tid == 0) left[atomicAdd(&counts->medium, 1u)] = entry;
            go_on();
            __syncthreads();
            continue;
        }
        // f(record) for every record that brought a key, by one thread
        auto for_each_key = [&](auto&& f)
        {
            #pragma unroll 1
            for(u32 t = tid; t < winners; t += BLOCK) f(u32(lines[CAP - 1 - t]));
            #pragma unroll 1
            for(u32 t = tid; t < open_ones; t += BLOCK) if(lines[t] & WON) f(u32(lines[t]) & RECORD);
        };
        for(u32 i = tid; i < (m + 7) / 8; i += BLOCK) reinterpret_cast<uint4*>(bin)[i] = make_uint4(0, 0, 0, 0);
        if(!PACKED)
            #pragma unroll 1
            for(u32 j = tid; j < m; j += BLOCK) sa[base + j] = SA_OPEN;         // suffixes that are alone go there later
        else
            #pragma unroll 1
            for(u32 j = tid; j < 5 * m; j += BLOCK) sa40[5 * u64(base) + j] = j % 5 < 4 ? u8(SA_OPEN) : u8(0);
        __syncthreads();
        for_each_key([&](const u32 e)
        {
            const u32 b = __umulhi(keys[e], m);
            atomicAdd(&bin[b >> 1], u32(cnt[e]) << (16 * (b & 1u)));
        });
        __syncthreads();
        // exclusive sums of the bins' counts, in place
        {
            u32 c[WORDS], sum = 0;
            const u32 w0 = tid * WORDS;
            const bool any = 2 * w0 < m;            // the words up to a multiple of four were cleared
            #pragma unroll
            for(u32 w = 0; w < WORDS; w += 4)
            {
                const uint4 v = any && 2 * (w0 + w) < m ? *reinterpret_cast<const uint4*>(bin + w0 + w) : make_uint4(0, 0, 0, 0);
                c[w] = v.x; c[w + 1] = v.y; c[w + 2] = v.z; c[w + 3] = v.w;
            }
            #pragma unroll
            for(u32 w = 0; w < WORDS; ++w) sum += (c[w] & 0xFFFFu) + (c[w] >> 16);
            const u32 inc = warp_inclusive(sum);
            if(lane == 31) warp_tot[tid >> 5] = inc;
            __syncthreads();
            u32 run = __reduce_add_sync(0xFFFFFFFFu, lane < (tid >> 5) ? warp_tot[lane] : 0u) + inc - sum;
            if(any)
            {
                #pragma unroll
                for(u32 w = 0; w < WORDS; ++w)
                {
                    bin[w0 + w] = run * 0x10001u + (c[w] << 16);        // below 2^16 each
                    run += (c[w] & 0xFFFFu) + (c[w] >> 16);
                }
            }
        }
        __syncthreads();
        // a key's place: behind the smaller ones of its list
        for_each_key([&](const u32 e)
        {
            const u32 key = keys[e], b = __umulhi(key, m);
            u32 place = start[b];
            for(u32 o = head[b]; o != NONE; o = link[o])
                if(keys[o] < key) place += cnt[o];
            res[e] = place | (res[e] & 0x7FFF0000u) | 1u << 31;
        });
        __syncthreads();
        for_each_key([&](const u32 e)
        {
            const u32 size = cnt[e];
            if(size > 1) link[e] = u16(atomicAdd(&s_tied[size <= SMALL_GROUP ? 0 : 1], size));
            if(size > NARROW_GROUP) s_wide = 1;
        });
        __syncthreads();
        const u32 small_ones = s_tied[0], all_ones = small_ones + s_tied[1];
        if(tid < 2)
        {
            const u32 c = s_tied[tid];
            s_slot[tid] = c ? atomicAdd(tid ? &counts->large : &counts->small, c) : 0;
        }
        for_each([&](const u32 i, const u32 j)
        {
            u32 e, number;
            if(open >> i & 1u)
            {
                const u32 x = res[j];
                e = x >> 31 ? j : x & 0xFFFFu;
                number = x >> 16 & 0x7FFFu;
            }
            else { e = key_of[i] & 0xFFFFu; number = key_of[i] >> 16; }
            const u32 first = res[e] & 0xFFFFu, size = cnt[e];
            if(size == 1) { put(base + first, p[i]); return; }
            const u32 o = link[e] + number + (size <= SMALL_GROUP ? 0u : small_ones);
            heads[o] = base + first;
            keys[o] = p[i];
        });
        __syncthreads();
        go_on();
        #pragma unroll 2
        for(u32 j = tid; j < all_ones; j += BLOCK)
        {
            const u64 e = u64(heads[j]) << 32 | keys[j];
            if(j < small_ones) list[u64(s_slot[0]) + j] = e;
            else list[list_cap - 1 - (u64(s_slot[1]) + (j - small_ones))] = e;
        }
        __syncthreads();        // the next batch reuses the shared arrays
    }
    if(tid == 0 && s_wide) counts->wide = 1;
}

// ---- what the kernels above leave -------------------------------------------------------------------------------------------------------

template <int BLOCK, int ITEMS> constexpr size_t LOCAL_SMEM = size_t(BLOCK * ITEMS) * 8 + (BLOCK * ITEMS / 2 + 8) * 4 + ((1 << MAX_B2) + 4) * 4;
constexpr u32 CROWDED_BIN = 8;      // a batch with larger bins is looked through for bins of one key
constexpr u32 MANY_TIED = 256;      // a batch with more tied records writes them to the list side by side
constexpr u32 LONG_BIN = 256;       // a bin of several keys with more records is not ordered by comparing all with all
static_assert(MEDIUM_CAP <= 8192, "slots of a batch take 13 bits");

// A record's place in its batch (13 bits), then the first place of its group or, where that is its own, the group's size (14 bits)
// and FIRST; SMALL or LARGE by the group's size, neither for a record that is alone.
constexpr u32 PL_SMALL = 1u << 27, PL_LARGE = 1u << 28, PL_FIRST = 1u << 29;
__device__ __forceinline__ u32 packed_place(const u32 place, const u32 head, const u32 size)
{
    return place | (place == head ? size << 13 | PL_FIRST : head << 13) | (size == 1 ? 0u : (size <= SMALL_GROUP ? PL_SMALL : PL_LARGE));
}

// The batch's entries [base, base + m) as 5-byte ones, from shared memory: four are 20 bytes, which begin on a word where the first's slot is a multiple of
// four; the words of 128 entries go out side by side by way of the warp's part of `words`. The up to three entries before and behind go byte by byte.
template <int BLOCK, int CAP>
__device__ __forceinline__ void write_packed(u32* words, const u32* placed, const u32 m, const u32 base, u8* __restrict__ sa40)
{
    constexpr u32 WARPS = BLOCK / 32;
    static_assert(CAP / WARPS >= 160, "a warp's words");
    const u32 tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const u32 head = min(m, (0u - base) & 3u), fours = (m - head) >> 2, tail = head + 4 * fours;
    u32* const mine = words + warp * (CAP / WARPS);
    u32* const out = reinterpret_cast<u32*>(sa40 + 5 * u64(base + head));
    for(u32 q0 = warp * 32; q0 < fours; q0 += WARPS * 32)
    {
        if(q0 + lane < fours)
        {
            const u32 e = head + 4 * (q0 + lane);
            const u32 a = placed[e], b = placed[e + 1], c = placed[e + 2], d = placed[e + 3];
            u32* const w = mine + 5 * lane;
            w[0] = a; w[1] = b << 8; w[2] = b >> 24 | c << 16; w[3] = c >> 16 | d << 24; w[4] = d >> 8;
        }
        __syncwarp();
        const u32 count = min(fours - q0, 32u) * 5;
        for(u32 k = lane; k < count; k += 32) out[u64(q0) * 5 + k] = mine[k];
        __syncwarp();
    }
    if(tid < (head + m - tail) * 5)
    {
        const u32 e = tid < head * 5 ? tid / 5 : tail + (tid - head * 5) / 5, byte = tid % 5;
        sa40[5 * u64(base + e) + byte] = byte < 4 ? u8(placed[e] >> (8 * byte)) : u8(0);
    }
}

// Single children of SORT_MOST to MEDIUM_CAP suffixes, and what the kernels above leave: one or two batches in ten thousand where symbols are independent, those with bins of more than SMALL_GROUP records
// or too many comparisons else. Every record is compared with all of its bin, of which there are as many as
// records; a bin of one key takes no comparisons, and a bin of many records of several keys sends the batch through a sorting network. The chain of its steps takes 20 us whatever there is to do.
// PACKED: the array is written to sa40 as 5-byte entries, else to sa.
template <int BLOCK, int ITEMS, int BLOCKS, bool PACKED>
__global__ void __launch_bounds__(BLOCK, BLOCKS) left_children_kernel(const u64* __restrict__ rec, const int bits, const u32* __restrict__ child_off, u32* __restrict__ sa, u8* __restrict__ sa40,
                                                                      u64* __restrict__ list, const u64 list_cap, Build_Counts* __restrict__ counts, const u32* __restrict__ left)
{
    constexpr int CAP = BLOCK * ITEMS;
    static_assert(ITEMS % 8 == 0, "a thread sums whole 16-byte pieces of the bins' counts");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u32* const keys = reinterpret_cast<u32*>(smem_raw);                             // [CAP]
    u32* const placed = keys + CAP;                                                 // [CAP] positions in their order
    u32* const bin = placed + CAP;                                                  // [CAP / 2 + 8]: two 16-bit counters a word, then the bins' starts
    u16* const start = reinterpret_cast<u16*>(bin);
    u32* const coff = bin + CAP / 2 + 8;                                            // [children of the batch + 1] their offsets
    __shared__ u32 warp_tot[BLOCK / 32];
    __shared__ u32 s_wide;
    __shared__ u32 s_tied[2], s_slot[2];            // records of small and of large groups in the batch, and their places in the list
    __shared__ u32 mixed[CAP / 32], s_crowded;      // a bit per bin: it holds several keys; whether any bin holds many records
    const u32 tid = threadIdx.x;
    const u32 children = 1u << bits;
    const int rbits = 32 - bits;                    // key bits behind the child's

    let_next_in();
    wait_for_previous();
    const u32 works = counts->medium;
    if(tid == 0) s_wide = 0;    // a barrier of the first batch comes before it is told
    for(u32 work = blockIdx.x; work < works; work += gridDim.x)
    {
        const u32 entry = left[work], child0 = entry >> MAX_B2, last = (entry & ((1u << MAX_B2) - 1)) + 1;
        const u32 first_digit = child0 & (children - 1);
        for(u32 d = tid; d <= last; d += BLOCK) coff[d] = __ldg(child_off + child0 + d);
        if(tid < 2) s_tied[tid] = 0;
        __syncthreads();
        u32 cur = 0;
        while(cur < last)
        {
            // a batch: as many children as fit
            u32 e = last;
            const u32 base = coff[cur];
            if(coff[e] - base > u32(CAP))
            {
                u32 a = cur, b = last;                  // the last e with coff[e] - base <= CAP
                while(b - a > 1)
                {
                    const u32 m = (a + b) >> 1;
                    if(coff[m] - base <= u32(CAP)) a = m; else b = m;
                }
                e = a;
                if(e == cur)            // no such child is left here
                {
                    ++cur;
                    continue;
                }
            }
            const u32 m = coff[e] - base;
            const bool single = e - cur == 1;
            cur = e;
            if(m == 0) continue;

            // Bins: a record's place inside its child by interpolation of its remaining key bits; there are as many bins as records.
            for(u32 i = tid; i < (m / 2 + 8) / 8 * 2; i += BLOCK) reinterpret_cast<uint4*>(bin)[i] = make_uint4(0, 0, 0, 0);
            if(tid < CAP / 32) mixed[tid] = 0;
            if(tid == 0) s_crowded = 0;
            u64 r[ITEMS];
            u32 pl[ITEMS];                      // bin << 16 | rank in the bin; of tied records later packed_place
            #pragma unroll
            for(int i = 0; i < ITEMS; ++i)
            {
                if(i * BLOCK >= m) break;       // of all threads: half of a full batch is the rule
                const u32 j = tid + i * BLOCK;
                if(j < m) r[i] = rec[base + j];
            }
            __syncthreads();
            #pragma unroll
            for(int i = 0; i < ITEMS; ++i)
            {
                if(i * BLOCK >= m) break;
                if(tid + i * BLOCK < m)
                {
                    const u32 k = u32(r[i] >> 32);
                    u32 b;
                    if(single) b = __umulhi(k << bits, m);
                    else
                    {
                        const u32 d = (bits ? k >> rbits : 0u) - first_digit, c0 = coff[d];
                        b = c0 - base + __umulhi(k << bits, coff[d + 1] - c0);
                    }
                    const u32 old = atomicAdd(&bin[b >> 1], (b & 1) ? 0x10000u : 1u);
                    pl[i] = (b << 16) | ((b & 1) ? old >> 16 : old & 0xFFFFu);
                }
            }
            __syncthreads();
            // exclusive sums of the bins' counts, in place; start[m] = m
            u32 longest = 0;        // of the even and of the odd bins
            {
                constexpr int WORDS = CAP / 2 / BLOCK;
                u32 c[WORDS], sum = 0;
                const u32 w0 = tid * WORDS;
                const bool any = 2 * w0 <= m;           // the words up to a multiple of WORDS were cleared
                if(any)
                {
                    #pragma unroll
                    for(int k = 0; k < WORDS / 4; ++k)
                    {
                        const uint4 v = reinterpret_cast<const uint4*>(bin)[tid * (WORDS / 4) + k];
                        c[4 * k] = v.x; c[4 * k + 1] = v.y; c[4 * k + 2] = v.z; c[4 * k + 3] = v.w;
                    }
                    u32 both = 0;           // two sums side by side: below 2^16 each
                    #pragma unroll
                    for(int k = 0; k < WORDS; ++k) { both += c[k]; longest = __vmaxu2(longest, c[k]); }
                    sum = (both & 0xFFFFu) + (both >> 16);
                }
                const u32 inc = warp_inclusive(sum);
                if(lane_id() == 31) warp_tot[tid >> 5] = inc;
                __syncthreads();
                u32 run = __reduce_add_sync(0xFFFFFFFFu, lane_id() < (tid >> 5) ? warp_tot[lane_id()] : 0u) + inc - sum;
                if(any)
                {
                    #pragma unroll
                    for(int k = 0; k < WORDS; ++k)
                    {
                        const u32 a = run * 0x10001u + (c[k] << 16);        // below 2^16 each
                        run += (c[k] & 0xFFFFu) + (c[k] >> 16);
                        c[k] = a;
                    }
                    #pragma unroll
                    for(int k = 0; k < WORDS / 4; ++k)
                        reinterpret_cast<uint4*>(bin)[tid * (WORDS / 4) + k] = make_uint4(c[4 * k], c[4 * k + 1], c[4 * k + 2], c[4 * k + 3]);
                }
            }
            if(m == u32(CAP) && tid == 0) start[CAP] = u16(CAP);       // behind the threads' words
            longest = max(longest & 0xFFFFu, longest >> 16);
            if(longest > CROWDED_BIN) s_crowded = 1;
            __syncthreads();
            u32 tied = 0;           // a bit per record
            // Only the keys are staged, in their bins; a record stays with its thread and counts the smaller and the equal keys of its bin.
            #pragma unroll
            for(int i = 0; i < ITEMS; ++i)
            {
                if(i * BLOCK >= m) break;
                if(tid + i * BLOCK < m) keys[start[pl[i] >> 16] + (pl[i] & 0xFFFFu)] = u32(r[i] >> 32);
            }
            __syncthreads();
            // Bins of many records are as a rule copies of one key (documents that occur many times): their places are known then.
            const bool crowded = s_crowded != 0;
            bool by_network = false;
            if(crowded)
            {
                #pragma unroll
                for(int i = 0; i < ITEMS; ++i)
                {
                    if(i * BLOCK >= m) break;
                    if(tid + i * BLOCK < m)
                    {
                        const u32 b = pl[i] >> 16, s = start[b];
                        if(keys[s] == u32(r[i] >> 32)) continue;
                        atomicOr(&mixed[b >> 5], 1u << (b & 31));
                        by_network |= start[b + 1] - s > LONG_BIN;
                    }
                }
                by_network = __syncthreads_or(by_network);
            }
            if(!by_network)
            {
                #pragma unroll
                for(int i = 0; i < ITEMS; ++i)
                {
                    if(i * BLOCK >= m) break;
                    if(tid + i * BLOCK < m)
                    {
                        const u32 k = u32(r[i] >> 32), b = pl[i] >> 16, s = start[b], t = start[b + 1];
                        u32 less = 0, upto = 0;
                        if(crowded && t - s > 1 && (mixed[b >> 5] >> (b & 31) & 1u) == 0)
                        {
                            const u32 place = s + (pl[i] & 0xFFFFu);
                            placed[place] = SA_OPEN;
                            pl[i] = packed_place(place, s, t - s);
                            tied |= 1u << i;
                            continue;
                        }
                        #pragma unroll
                        for(u32 j = 0; j < 4; ++j)      // most bins hold no more: four reads in flight
                            if(s + j < t) { const u32 o = keys[s + j]; less += o < k; upto += o <= k; }
                        for(u32 j = s + 4; j < t; ++j) { const u32 o = keys[j]; less += o < k; upto += o <= k; }
                        const u32 head = s + less;
                        if(upto - less == 1) placed[head] = u32(r[i]);
                        else
                        {
                            const u32 mine = s + (pl[i] & 0xFFFFu);
                            u32 place = head;
                            for(u32 j = s; j < mine; ++j) place += keys[j] == k;
                            placed[place] = SA_OPEN;
                            pl[i] = packed_place(place, head, upto - less);
                            tied |= 1u << i;
                        }
                    }
                }
            }
            else
            {
                // Many records of several keys in one bin: a sorting network over the batch (keys and positions), then every record finds its
                // group's ends by bisection.
                u32 size = 1;
                while(size < m) size <<= 1;
                #pragma unroll
                for(int i = 0; i < ITEMS; ++i)
                {
                    const u32 j = tid + i * BLOCK;
                    if(j >= size) break;
                    keys[j] = j < m ? u32(r[i] >> 32) : 0xFFFFFFFFu;
                    placed[j] = j < m ? u32(r[i]) : 0xFFFFFFFFu;        // no position: behind all records
                }
                __syncthreads();
                for(u32 k = 2; k <= size; k <<= 1)
                    for(u32 d = k >> 1; d > 0; d >>= 1)
                    {
                        for(u32 t = tid; t < size / 2; t += BLOCK)
                        {
                            const u32 a = 2 * t - (t & (d - 1)), b = a + d;
                            const u32 x = keys[a], y = keys[b], px = placed[a], py = placed[b];
                            if((x > y || (x == y && px > py)) == ((a & k) == 0)) { keys[a] = y; keys[b] = x; placed[a] = py; placed[b] = px; }
                        }
                        __syncthreads();
                    }
                #pragma unroll
                for(int i = 0; i < ITEMS; ++i)
                {
                    const u32 j = tid + i * BLOCK;
                    if(j >= m) break;
                    const u32 key = keys[j];
                    r[i] = placed[j];
                    u32 a = 0, b = j;                   // first record with this key
                    while(a < b) { const u32 mid = (a + b) >> 1; if(keys[mid] < key) a = mid + 1; else b = mid; }
                    u32 c = j + 1, f = m;               // first record behind with a greater key
                    while(c < f) { const u32 mid = (c + f) >> 1; if(keys[mid] <= key) c = mid + 1; else f = mid; }
                    if(c - a == 1) continue;
                    placed[j] = SA_OPEN;
                    pl[i] = packed_place(j, a, c - a);
                    tied |= 1u << i;
                }
            }
            const bool ties = __syncthreads_or(tied != 0);
            if(PACKED) write_packed<BLOCK, CAP>(keys, placed, m, base, sa40);
            else
            {
                #pragma unroll
                for(int i = 0; i < ITEMS; ++i)
                {
                    const u32 j = tid + i * BLOCK;
                    if(j >= m) break;
                    sa[base + j] = placed[j];
                }
            }
            // The tied records go to the list, a group's side by side: the first of a group takes its places (start[] is free now).
            if(ties)
            {
                if(tied)            // a few threads of a block as a rule
                {
                    #pragma unroll
                    for(int i = 0; i < ITEMS; ++i)
                        if((tied >> i & 1u) && (pl[i] & PL_FIRST))
                        {
                            const u32 size = pl[i] >> 13 & 16383u;
                            start[pl[i] & 8191u] = u16(atomicAdd(&s_tied[(pl[i] & PL_SMALL) ? 0 : 1], size));
                            if(size > NARROW_GROUP) s_wide = 1;
                        }
                }
                __syncthreads();
                const u32 small_ones = s_tied[0], all_ones = small_ones + s_tied[1];
                const bool many = all_ones > MANY_TIED;     // by way of shared memory (keys and placed are free now), side by side
                __syncthreads();
                if(tid < 2)
                {
                    const u32 c = s_tied[tid];
                    s_slot[tid] = c ? atomicAdd(tid ? &counts->large : &counts->small, c) : 0;
                    s_tied[tid] = 0;
                }
                if(!many) __syncthreads();
                if(tied)
                {
                    #pragma unroll
                    for(int i = 0; i < ITEMS; ++i)
                        if(tied >> i & 1u)
                        {
                            const u32 place = pl[i] & 8191u, head = (pl[i] & PL_FIRST) ? place : pl[i] >> 13 & 8191u;
                            const bool small = (pl[i] & PL_SMALL) != 0;
                            const u32 at = start[head] + (place - head);
                            if(many)
                            {
                                const u32 k = small ? at : small_ones + at;
                                keys[k] = base + head;
                                placed[k] = u32(r[i]);
                                continue;
                            }
                            const u64 k = u64(s_slot[small ? 0 : 1]) + at;
                            list[small ? k : list_cap - 1 - k] = (u64(base + head) << 32) | u32(r[i]);
                        }
                }
                if(many)
                {
                    __syncthreads();
                    for(u32 j = tid; j < all_ones; j += BLOCK)
                    {
                        const u64 e = (u64(keys[j]) << 32) | placed[j];
                        if(j < small_ones) list[u64(s_slot[0]) + j] = e;
                        else list[list_cap - 1 - (u64(s_slot[1]) + (j - small_ones))] = e;
                    }
                }
            }
            __syncthreads();        // the next batch reuses the shared arrays
        }
        __syncthreads();            // a run may end in an empty child: coff is still being read then
    }
    if(tid == 0 && s_wide) counts->wide = 1;
}

// Every oversize child is copied by the blocks of one grid row (blockIdx.y): keys = (first slot << 32) | key, vals = position.
__global__ void __launch_bounds__(256) gather_oversize_kernel(const u64* __restrict__ rec, const u32* __restrict__ over, const u32 oversize, const u32* __restrict__ child_off,
                                                             u64* __restrict__ keys, u32* __restrict__ vals, u32* __restrict__ cursor)
{
    __shared__ u32 s_at;
    for(u32 o = blockIdx.y; o < oversize; o += gridDim.y)
    {
        const u32 first = child_off[over[o]], end = child_off[over[o] + 1];
        for(u64 b = u64(first) + u64(blockIdx.x) * 2048; b < end; b += u64(gridDim.x) * 2048)
        {
            const u32 c = end - b < 2048 ? u32(end - b) : 2048u;
            if(threadIdx.x == 0) s_at = atomicAdd(cursor, c);
            __syncthreads();
            for(u32 j = threadIdx.x; j < c; j += 256)
            {
                const u64 v = rec[b + j];
                keys[s_at + j] = (u64(first) << 32) | (v >> 32);
                vals[s_at + j] = u32(v);
            }
            __syncthreads();
        }
    }
}

// The entries of oversize children from sa to sa40.
__global__ void __launch_bounds__(256) pack_oversize_kernel(const u32* __restrict__ sa, const u32* __restrict__ over, const u32 oversize, const u32* __restrict__ child_off,
                                                           u8* __restrict__ sa40)
{
    for(u32 o = blockIdx.y; o < oversize; o += gridDim.y)
    {
        const u64 first = u64(child_off[over[o]]) * 5, end = u64(child_off[over[o] + 1]) * 5;
        for(u64 b = first + u64(blockIdx.x) * 256 + threadIdx.x; b < end; b += u64(gridDim.x) * 256)
        {
            const u32 byte = u32(b % 5);
            sa40[b] = byte < 4 ? u8(sa[b / 5] >> (8 * byte)) : u8(0);
        }
    }
}

template <typename K>
int shared_bytes(csa_ctx* ctx, K kern, size_t bytes, std::atomic<bool>* configured)
{
    if(!configured[ctx->device & 63])
    {
        CSA_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
        configured[ctx->device & 63] = true;
    }
    return CSA_OK;
}

template <int BLOCK, bool PART>
int launch_scatter_text(csa_ctx* ctx, const u16* T, u64 n, const u32* code, int bits, int keep_top, u32 first_bin, u32 part_bins, u32* cursor, u64* out)
{
    static std::atomic<bool> configured[64];
    CSA_TRY(shared_bytes(ctx, scatter_text_kernel<BLOCK, PART>, SCATTER_TEXT_SMEM<BLOCK>, configured));
    launch_early(scatter_text_kernel<BLOCK, PART>, unsigned(div_up(n, TILE_POSITIONS<BLOCK>)), BLOCK, SCATTER_TEXT_SMEM<BLOCK>, ctx->stream, T, n, code, bits, keep_top, first_bin, part_bins, cursor, out);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

// Small texts take small tiles, so that every SM gets one. From 2^19 suffixes on 65 wide tiles do better than 265 small ones, which make as many global atomics each: 6e5 tokens 157 -> 140 us a build, 1e6
// 185 -> 146, 2e6 246 -> 170, 4e6 near-duplicates 1276 -> 1200; at 3e5 there is no difference.
bool wide_tiles(u64 n) { return n >= (u64(1) << 19); }

}   // namespace

Prefix_Sort prefix_sort_plan(u64 n)
{
    Prefix_Sort ps;
    ps.n = n;
    // Children of at most 2048 suffixes on average. Between 2^21 and 2^26 suffixes, 1536: a child that the local sort leaves to its second kernel, one in a thousand at 2048, costs 20 us wherever
    // that one ends (2^24 tokens 502 -> 490 us, 8e6 315 -> 299); above, runs of twice as many records in the second split are worth more (1.25e8 tokens 2.44 ms against 2.40).
    int t = 0;
    while(t < MAX_B1 && (n >> t) > 2048) ++t;
    if((n >> t) > 2048)
        while(t < MAX_B1 + MAX_B2 && (n >> t) > (n < (u64(1) << 26) ? 1536 : 2048)) ++t;
    ps.b1 = t <= MAX_B1 ? 0 : t / 2;
    ps.b2 = t - ps.b1;
    ps.key_bits = ps.b1 + 32;
    ps.parents = 1u << ps.b1;
    ps.children = 1u << ps.b2;
    return ps;
}

size_t prefix_sort_table_bytes(const Prefix_Sort& ps)
{
    const u64 all = u64(ps.parents) * ps.children;
    return align_up256(65536 * 4) * 2 + align_up256((size_t(1) << MAX_B1) * 4 + 4) * 4 + align_up256(all * 4) * 3 + align_up256((all + 1) * 4) + align_up256(most_batches(ps.parents, ps.children) * sizeof(uint4)) + 4096;
}

bool prefix_sort_carve(Carver& cv, const Prefix_Sort& ps, Prefix_Tables& t)
{
    const u64 all = u64(ps.parents) * ps.children;
    t.hist = cv.take<u32>(65536);
    t.cnt1 = cv.take<u32>(size_t(1) << MAX_B1);
    t.code = cv.take<u32>(65536);
    t.cur1 = cv.take<u32>(size_t(1) << MAX_B1);
    t.par_off = cv.take<u32>((size_t(1) << MAX_B1) + 1);
    t.tile0 = cv.take<u32>((size_t(1) << MAX_B1) + 1);
    t.cnt2 = cv.take<u32>(all);
    t.child_off = cv.take<u32>(all + 1);
    t.over = cv.take<u32>(all);
    t.left = cv.take<u32>(all);
    t.batches = cv.take<uint4>(most_batches(ps.parents, ps.children));
    return cv.ok;
}

namespace
{

// The code of the text's symbols; the counters of the first split, of the build and of `children` children are cleared on the way.
int launch_code(csa_ctx* ctx, const Prefix_Tables& t, const u16* T, const u64 n, Build_Counts* counts, const u32 children)
{
    // the code, from every symbol of a small text or a million of a large one
    static_assert(CODE_BLOCK == 1 << MAX_B1, "block 0 of make_code_kernel clears a counter of the first split per thread");
    if(n <= CODE_COUNT_MAX)
    {
        static std::atomic<bool> configured[64];
        CSA_TRY(shared_bytes(ctx, make_code_kernel<true>, CODE_SMEM, configured));
        make_code_kernel<true><<<65536 / CODE_WALKERS, CODE_BLOCK, CODE_SMEM, ctx->stream>>>(T, u32(n), nullptr, u32((u64(1) << 22) / n), t.code, t.cnt1, reinterpret_cast<u32*>(counts), t.cnt2, children);
        CSA_LAUNCH_CHECK(ctx);
    }
    else
    {
        static std::atomic<bool> configured[2][64];
        CSA_TRY(shared_bytes(ctx, sample_symbols_kernel, HIST_SMEM, configured[0]));
        CSA_TRY(shared_bytes(ctx, make_code_kernel<false>, CODE_SMEM, configured[1]));
        const u64 pieces = n / 8, vectors = pieces < (u64(1) << 17) ? pieces : (u64(1) << 17);
        const u64 samples = vectors == pieces ? n : vectors * 8;
        const u64 blocks = div_up(vectors, HIST_BLOCK);
        CSA_CUDA(ctx, cudaMemsetAsync(t.hist, 0, 65536 * 4, ctx->stream));
        sample_symbols_kernel<<<unsigned(blocks > 148 ? 148 : blocks), HIST_BLOCK, HIST_SMEM, ctx->stream>>>(T, n, vectors, t.hist);
        CSA_LAUNCH_CHECK(ctx);
        launch_early(make_code_kernel<false>, 65536 / CODE_WALKERS, CODE_BLOCK, CODE_SMEM, ctx->stream, T, u32(n), t.hist, u32((u64(1) << 22) / samples), t.code, t.cnt1,
                     reinterpret_cast<u32*>(counts), t.cnt2, children);
        CSA_LAUNCH_CHECK(ctx);
    }
    return CSA_OK;
}

int launch_count_text(csa_ctx* ctx, const u16* T, u64 n, const u32* code, int bits, u32* counts)
{
    if(wide_tiles(n))
    {
        static std::atomic<bool> configured[64];
        CSA_TRY(shared_bytes(ctx, count_long_text_kernel, COUNT_SMEM, configured));
        count_long_text_kernel<<<148, COUNT_BLOCK, COUNT_SMEM, ctx->stream>>>(T, n, code, bits, counts);
    }
    else launch_early(count_text_kernel<128>, unsigned(div_up(n, TILE_POSITIONS<128>)), 128, 0, ctx->stream, T, n, code, bits, counts);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

// The three are let in early, one behind the other (2^24 tokens 465 -> 456 us a build, 3e6 217 -> 211), and make_code_kernel has cleared the counters, so that no other work of the stream lies between.
template <int BLOCK>
int launch_split_kernels(csa_ctx* ctx, const Prefix_Tables& t, u32 parents, int b2, u64 n, const u64* recA, u64* recB, Build_Counts* counts)
{
    const unsigned tiles = unsigned(n / (BLOCK * SPLIT_ITEMS) + parents);
    const u32 children = 1u << b2;
    launch_early(count_children_kernel<BLOCK>, tiles, BLOCK, 0, ctx->stream, recA, t.par_off, t.tile0, parents, b2, t.cnt2);
    CSA_LAUNCH_CHECK(ctx);
    launch_early(child_offsets_kernel, parents, 1024, 0, ctx->stream, t.cnt2, t.par_off, parents, children, t.child_off, t.batches, t.over, t.left, counts);
    CSA_LAUNCH_CHECK(ctx);
    static std::atomic<bool> configured[64];
    CSA_TRY(shared_bytes(ctx, scatter_children_kernel<BLOCK>, SPLIT_SMEM<BLOCK>, configured));
    launch_early(scatter_children_kernel<BLOCK>, tiles, BLOCK, SPLIT_SMEM<BLOCK>, ctx->stream, recA, t.par_off, t.tile0, parents, b2, t.cnt2, recB);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

// The second split of `parents` buckets with n records in all (recA to recB); the children's counters (cnt2) are cleared.
int launch_second_split(csa_ctx* ctx, const Prefix_Tables& t, u32 parents, int b2, u64 n, const u64* recA, u64* recB, Build_Counts* counts)
{
    return split_block(b2) == 1024 ? launch_split_kernels<1024>(ctx, t, parents, b2, n, recA, recB, counts) : launch_split_kernels<512>(ctx, t, parents, b2, n, recA, recB, counts);
}

// The second launch takes batches of many copies, the third what else the ones before leave: little or nothing as a rule, so their blocks are let in early.
template <bool PACKED>
int launch_local_sort(csa_ctx* ctx, const Prefix_Tables& t, u32 parents, int b2, u64 n, const u64* rec, u32* sa, u8* sa40, u64* list, Build_Counts* counts)
{
    const u32 over_cap = parents << b2;
    const bool crowds = parents > 1;        // a text of one split goes to the third kernel with what it leaves: a launch counts there, and 1e6 near-duplicates take as long either way
    static std::atomic<bool> configured[3][64];
    CSA_TRY(shared_bytes(ctx, local_sort_kernel<PACKED>, SORT_SMEM<PACKED>, configured[0]));
    CSA_TRY(shared_bytes(ctx, crowded_batches_kernel<PACKED>, CROWD_SMEM, configured[1]));
    CSA_TRY(shared_bytes(ctx, left_children_kernel<512, 16, 2, PACKED>, LOCAL_SMEM<512, 16>, configured[2]));
    launch_early(local_sort_kernel<PACKED>, unsigned(std::min<u64>(over_cap, SORT_GRID)), SORT_BLOCK, SORT_SMEM<PACKED>, ctx->stream, rec, t.batches, b2, sa, sa40, list, counts, t.over, crowds ? over_cap : 0u, t.left);
    CSA_LAUNCH_CHECK(ctx);
    if(crowds)
    {
        launch_early(crowded_batches_kernel<PACKED>, 148 * 3, CROWD_BLOCK, CROWD_SMEM, ctx->stream, rec, b2, t.child_off, sa, sa40, list, n, counts, t.over, over_cap, t.left);
        CSA_LAUNCH_CHECK(ctx);
    }
    launch_early(left_children_kernel<512, 16, 2, PACKED>, LEFT_BLOCKS, 512, LOCAL_SMEM<512, 16>, ctx->stream, rec, b2, t.child_off, sa, sa40, list, n, counts, t.left);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

}   // namespace

int launch_prefix_sort(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, u64* recA, u64* recB, u32* sa, u8* sa40, u32 p, Build_Counts* counts,
                       u64** list, u64** records, cudaEvent_t after_first_split)
{
    const u64 n = ps.n;
    CSA_TRY(launch_code(ctx, t, T, n, counts, ps.b1 ? ps.parents << ps.b2 : 0u));
    const bool one_level = ps.b1 == 0;
    const int bits = one_level ? ps.b2 : ps.b1;
    if(bits > 0) CSA_TRY(launch_count_text(ctx, T, n, t.code, bits, t.cnt1));
    launch_early(parent_offsets_kernel, 1, 1024, 0, ctx->stream, t.cnt1, 1u << bits, u32(n), one_level ? 1 : 0, t.cur1, t.par_off, t.tile0, t.child_off, t.batches, t.over, t.left, u32(split_block(ps.b2) * SPLIT_ITEMS), p, counts);
    CSA_LAUNCH_CHECK(ctx);
    CSA_TRY(wide_tiles(n) ? (launch_scatter_text<512, false>(ctx, T, n, t.code, bits, one_level ? 1 : 0, 0, 0, t.cur1, recA))
                          : (launch_scatter_text<128, false>(ctx, T, n, t.code, bits, one_level ? 1 : 0, 0, 0, t.cur1, recA)));
    CSA_CUDA(ctx, cudaEventRecord(after_first_split, ctx->stream));
    ctx->counters[1] += one_level ? 1 : 2;
    ctx->counters[2] += one_level ? n : 2 * n;
    u64* rec = recA;
    u64* other = recB;
    if(!one_level)
    {
        CSA_TRY(launch_second_split(ctx, t, ps.parents, ps.b2, n, recA, recB, counts));
        rec = recB; other = recA;
    }
    CSA_TRY(sa ? launch_local_sort<false>(ctx, t, ps.parents, ps.b2, n, rec, sa, nullptr, other, counts)
               : launch_local_sort<true>(ctx, t, ps.parents, ps.b2, n, rec, nullptr, sa40, other, counts));
    *list = other;
    *records = rec;
    return CSA_OK;
}

Prefix_Sort prefix_sort_part_plan(u64 n)
{
    Prefix_Sort ps = prefix_sort_plan(n);
    const int t = ps.b1 + ps.b2;
    ps.b1 = t - 1 < 1 ? 1 : (t - 1 > MAX_B1 ? MAX_B1 : t - 1);
    ps.b2 = t - ps.b1 < 1 ? 1 : t - ps.b1;
    ps.key_bits = ps.b1 + 32;
    ps.parents = 1u << ps.b1;
    ps.children = 1u << ps.b2;
    return ps;
}

int launch_prefix_counts(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, Build_Counts* counts)
{
    CSA_TRY(launch_code(ctx, t, T, ps.n, counts, 0));
    return launch_count_text(ctx, T, ps.n, t.code, ps.b1, t.cnt1);
}

int launch_prefix_sort_part(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, u32 first_bin, u32 bins, u64 size, u64* recA, u64* recB, u32* sa,
                            Build_Counts* counts)
{
    CSA_CUDA(ctx, cudaMemsetAsync(counts, 0, sizeof(Build_Counts), ctx->stream));
    parent_offsets_kernel<<<1, 1024, 0, ctx->stream>>>(t.cnt1 + first_bin, bins, u32(size), 0, t.cur1, t.par_off, t.tile0, t.child_off, t.batches, t.over, t.left, u32(split_block(ps.b2) * SPLIT_ITEMS), 1, counts);
    CSA_LAUNCH_CHECK(ctx);
    CSA_TRY(wide_tiles(ps.n) ? (launch_scatter_text<512, true>(ctx, T, ps.n, t.code, ps.b1, 0, first_bin, bins, t.cur1, recA))
                             : (launch_scatter_text<128, true>(ctx, T, ps.n, t.code, ps.b1, 0, first_bin, bins, t.cur1, recA)));
    CSA_CUDA(ctx, cudaMemsetAsync(t.cnt2, 0, (size_t(bins) << ps.b2) * 4, ctx->stream));
    CSA_TRY(launch_second_split(ctx, t, bins, ps.b2, size, recA, recB, counts));
    CSA_TRY(launch_local_sort<false>(ctx, t, bins, ps.b2, size, recB, sa, nullptr, recA, counts));
    ctx->counters[1] += 2;
    ctx->counters[2] += 2 * size;
    return CSA_OK;
}

int launch_gather_oversize(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, u32 oversize, const u64* records, u64* keys, u32* vals, u32* cursor)
{
    (void)ps;
    if(oversize == 0) return CSA_OK;
    CSA_CUDA(ctx, cudaMemsetAsync(cursor, 0, 4, ctx->stream));
    // Few children are large ones as a rule (one symbol repeated: a single child): they get as many more blocks. With 32 for each, a child of
    // 2^24 suffixes took 1.2 ms; this way 0.06 ms.
    const unsigned rows = oversize < 1024 ? oversize : 1024;
    gather_oversize_kernel<<<dim3(std::max(32u, std::min(148u * 8, (1u << 14) / rows)), rows), 256, 0, ctx->stream>>>(records, t.over, oversize, t.child_off, keys, vals, cursor);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_pack_oversize(csa_ctx* ctx, const Prefix_Tables& t, u32 oversize, const u32* sa, u8* sa40)
{
    if(oversize == 0) return CSA_OK;
    const unsigned rows = oversize < 1024 ? oversize : 1024;
    pack_oversize_kernel<<<dim3(std::max(32u, std::min(148u * 8, (1u << 14) / rows)), rows), 256, 0, ctx->stream>>>(sa, t.over, oversize, t.child_off, sa40);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}
