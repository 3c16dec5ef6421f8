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
constexpr int SPLIT_BLOCK = 512, SPLIT_ITEMS = 16, SPLIT_TILE = SPLIT_BLOCK * SPLIT_ITEMS;
// Children that start inside one chunk of slots belong to one block: one child as a rule.
constexpr u32 LOCAL_CHUNK = 2048, SHORT_CHUNK = 1024;

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
                                                              u32* __restrict__ cnt1, u32* __restrict__ counts)
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

// Child `next - 1` occupies the slots [r0, r1) of its parent: the chunks that begin behind its start begin with the next child.
__device__ __forceinline__ void first_children(u32* __restrict__ chunk_first, const u32 chunks, const u32 chunk, const u32 r0, const u32 r1, const u32 next)
{
    for(u32 k = r0 / chunk + 1; k <= r1 / chunk && k < chunks; ++k) chunk_first[k] = next;
}

// Offsets of the parents and the work lists that follow from their sizes. one_level: there is no second split, the bins are
// the children of one parent that holds everything.
__global__ void __launch_bounds__(1024) parent_offsets_kernel(const u32* __restrict__ counts, const u32 bins, const u32 n, const int one_level, u32* __restrict__ cursor,
                                                             u32* __restrict__ par_off, u32* __restrict__ tile0, u32* __restrict__ chunk0, u32* __restrict__ child_off, u32* __restrict__ chunk_first,
                                                             const u32 p, Build_Counts* __restrict__ stats)
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
        const u32 chunks = (n + SHORT_CHUNK - 1) / SHORT_CHUNK;
        if(t < bins) { child_off[t] = off; first_children(chunk_first, chunks, SHORT_CHUNK, off, off + c, t + 1); }
        if(t == 0) { child_off[bins] = n; chunk0[1] = chunks; chunk_first[0] = 0; chunk_first[chunks] = bins; }
        return;
    }
    const u32 tiles = (c + SPLIT_TILE - 1) / SPLIT_TILE, chunks = (c + LOCAL_CHUNK - 1) / LOCAL_CHUNK;
    u32 all_tiles, all_chunks;
    const u32 t0 = block_exclusive<1024>(tiles, warp_tot, all_tiles);
    const u32 c0 = block_exclusive<1024>(chunks, warp_tot, all_chunks);
    if(t < bins) { par_off[t] = off; tile0[t] = t0; chunk0[t] = c0; }
    if(t == 0) { par_off[bins] = n; tile0[bins] = all_tiles; chunk0[bins] = all_chunks; }
}

template <int BLOCK> constexpr size_t SCATTER_TEXT_SMEM = size_t(TILE_POSITIONS<BLOCK>) * 8;
static_assert(SCATTER_TEXT_SMEM<512> >= sizeof(Tile_Code<512>) && SCATTER_TEXT_SMEM<128> >= sizeof(Tile_Code<128>), "the windows lie where the records are staged later");

// Scatter by the top `bits` bits: the places inside a bucket come from shared-memory atomics and, for the tile's run of a bucket,
// from one global atomic (the order inside a bucket is free); records are staged in bucket order and written as runs. What bounds it is shared memory
// and L1 (78 % of their wavefronts): so a staged record carries its bin and its place in the tile in one word instead of its position and a bin beside it.
// keep_top: the record keeps the top bits (there is no second split), else its key starts behind them. PART: only the suffixes of the
// buckets [first_bin, first_bin + part_bins) are taken, and the cursors are theirs.
template <int BLOCK, bool PART>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) scatter_text_kernel(const u16* __restrict__ T, const u64 n, const u32* __restrict__ code, const int bits,
                                                                          const int keep_top, const u32 first_bin, const u32 part_bins, u32* __restrict__ cursor,
                                                                          u64* __restrict__ out)
{
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
    u32 mine[PER], sum = 0;
    #pragma unroll
    for(int k = 0; k < PER; ++k) { const u32 b = threadIdx.x * PER + k; mine[k] = b < bins ? cnt[b] : 0; sum += mine[k]; }
    u32 total;
    u32 run = block_exclusive<BLOCK>(sum, warp_tot, total);
    #pragma unroll
    for(int k = 0; k < PER; ++k)
    {
        const u32 b = threadIdx.x * PER + k;
        if(b < bins)
        {
            cnt[b] = run;
            if(mine[k]) base[b] = atomicAdd(&cursor[b], mine[k]) - run;
        }
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

__global__ void __launch_bounds__(SPLIT_BLOCK) count_children_kernel(const u64* __restrict__ rec, const u32* __restrict__ par_off, const u32* __restrict__ tile0,
                                                                    const u32 parents, const int bits, u32* __restrict__ counts)
{
    __shared__ u32 cnt[1 << MAX_B2];
    __shared__ u32 found;
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

// One block per parent: the children's counts become their places (in counts, running) and their offsets (child_off).
__global__ void __launch_bounds__(1024) child_offsets_kernel(u32* __restrict__ counts, const u32* __restrict__ par_off, const u32 parents, const u32 children,
                                                            u32* __restrict__ child_off, const u32* __restrict__ chunk0, u32* __restrict__ chunk_first)
{
    __shared__ u32 warp_tot[32];
    const u32 p = blockIdx.x, t = threadIdx.x;
    u32* const c = counts + u64(p) * children;
    const u32 i0 = 2 * t, i1 = 2 * t + 1;          // up to 2048 children
    const u32 a = i0 < children ? c[i0] : 0, b = i1 < children ? c[i1] : 0;
    u32 total;
    const u32 rel = block_exclusive<1024>(a + b, warp_tot, total), off = par_off[p] + rel;
    const u32 chunks = chunk0[p + 1] - chunk0[p];
    if(i0 < children) first_children(chunk_first + chunk0[p], chunks, LOCAL_CHUNK, rel, rel + a, p * children + i0 + 1);
    if(i1 < children) first_children(chunk_first + chunk0[p], chunks, LOCAL_CHUNK, rel + a, rel + a + b, p * children + i1 + 1);
    if(t == 0 && chunks) chunk_first[chunk0[p]] = p * children;
    if(i0 < children) { c[i0] = off; child_off[u64(p) * children + i0] = off; }
    if(i1 < children) { c[i1] = off + a; child_off[u64(p) * children + i1] = off + a; }
    if(p == parents - 1 && t == 0) { child_off[u64(parents) * children] = par_off[parents]; chunk_first[chunk0[parents]] = parents * children; }
}

constexpr size_t SPLIT_SMEM = size_t(SPLIT_TILE) * 8;

__global__ void __launch_bounds__(SPLIT_BLOCK, 2) scatter_children_kernel(const u64* __restrict__ rec, const u32* __restrict__ par_off, const u32* __restrict__ tile0,
                                                                         const u32 parents, const int bits, u32* __restrict__ cursor, u64* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u64* const stage = reinterpret_cast<u64*>(smem_raw);
    __shared__ u32 cnt[1 << MAX_B2];
    __shared__ u32 base[1 << MAX_B2];
    __shared__ u32 warp_tot[SPLIT_BLOCK / 32];
    __shared__ u32 found;
    const u32 children = 1u << bits;
    for(u32 i = threadIdx.x; i < children; i += SPLIT_BLOCK) cnt[i] = 0;
    const u32 p = parent_of_block(tile0, parents, blockIdx.x, &found);
    if(p >= parents) return;
    const u32 end = par_off[p + 1], first = par_off[p] + (blockIdx.x - tile0[p]) * SPLIT_TILE;
    const u32 valid = end - first < u32(SPLIT_TILE) ? end - first : u32(SPLIT_TILE);
    u64 r[SPLIT_ITEMS];
    u32 place2[SPLIT_ITEMS / 2];         // ranks below 8192, two a register
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
    u32 mine[PER], sum = 0;
    #pragma unroll
    for(int k = 0; k < PER; ++k) { const u32 b = threadIdx.x * PER + k; mine[k] = b < children ? cnt[b] : 0; sum += mine[k]; }
    u32 total;
    u32 run = block_exclusive<SPLIT_BLOCK>(sum, warp_tot, total);
    #pragma unroll
    for(int k = 0; k < PER; ++k)
    {
        const u32 b = threadIdx.x * PER + k;
        if(b < children)
        {
            cnt[b] = run;
            if(mine[k]) base[b] = atomicAdd(&cursor[u64(p) * children + b], mine[k]) - run;
        }
        run += mine[k];
    }
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < SPLIT_ITEMS; ++i)
        if(threadIdx.x + i * SPLIT_BLOCK < valid)
            stage[cnt[u32(r[i] >> 32) >> (32 - bits)] + ((place2[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu)] = r[i];
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

template <int BLOCK, int ITEMS> constexpr size_t LOCAL_SMEM = size_t(BLOCK * ITEMS) * 8 + (BLOCK * ITEMS / 2 + 8) * 4 + ((1 << MAX_B2) + 4) * 4;
constexpr u32 MEDIUM_CAP = 512 * 16;        // records of the largest child that a block holds
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
            const u32* const v = placed + head + 4 * (q0 + lane);
            const u32 a = v[0], b = v[1], c = v[2], d = v[3];
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

// What bounds it is the issue of instructions (7 a record and warp, 68 % of the cycles), then barriers between dependent steps; memory is not (12 bytes a
// record). So a block finds its children in two dependent reads (chunk_first, child_off), records stay with their threads and only keys are staged,
// what only tied records need is skipped by warps without any, and three blocks of 512 threads with up to 8 records each share an SM (two such blocks
// 4.70 ms a build of 2e8 tokens, three 4.67 and with shorter sums of the bins 4.55; blocks of 256 with 16 records, four to an SM, 5.51, with 8 records 4.75; every record staged
// whole and looked up again by its place 5.17). A block reads its next chunk ahead.
// MEDIUM: the work list is `over` from its back, single children that were too large for the smaller block; else such children go
// there if a block of 16 records a thread holds them, and to the front, for the radix sort, if not.
// PACKED: the array is written to sa40 as 5-byte entries, else to sa.
template <int BLOCK, int ITEMS, int BLOCKS, bool MEDIUM, bool PACKED>
__global__ void __launch_bounds__(BLOCK, BLOCKS) local_sort_kernel(const u64* __restrict__ rec, const u32* __restrict__ chunk_first, const u32* __restrict__ chunks,
                                                                   const int bits, const u32* __restrict__ child_off, u32* __restrict__ sa, u8* __restrict__ sa40, u64* __restrict__ list,
                                                                   const u64 list_cap, Build_Counts* __restrict__ counts, u32* __restrict__ over, const u32 over_cap)
{
    constexpr int CAP = BLOCK * ITEMS;
    static_assert(ITEMS % 8 == 0, "a thread sums whole 16-byte pieces of the bins' counts");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u32* const keys = reinterpret_cast<u32*>(smem_raw);                             // [CAP]
    u32* const placed = keys + CAP;                                                 // [CAP] positions in their order
    u32* const bin = placed + CAP;                                                  // [CAP / 2 + 8]: two 16-bit counters a word, then the bins' starts
    u16* const start = reinterpret_cast<u16*>(bin);
    u32* const coff = bin + CAP / 2 + 8;                                            // [children of the chunk + 1] their offsets
    __shared__ u32 warp_tot[BLOCK / 32];
    __shared__ u32 s_tied[2], s_slot[2];            // records of small and of large groups in the batch, and their places in the list
    __shared__ u32 mixed[CAP / 32], s_crowded;      // a bit per bin: it holds several keys; whether any bin holds many records
    const u32 tid = threadIdx.x;
    const u32 children = 1u << bits;
    const int rbits = 32 - bits;                    // key bits behind the child's

    const u32 works = MEDIUM ? counts->medium : *chunks;
    u32 next_first = 0, next_end = 0;       // the children of the chunk after this one, read ahead
    auto look_up = [&](const u32 w)
    {
        next_first = MEDIUM ? over[over_cap - 1 - w] : __ldg(chunk_first + w);
        next_end = MEDIUM ? next_first + 1 : __ldg(chunk_first + w + 1);
    };
    if(blockIdx.x < works) look_up(blockIdx.x);
    for(u32 work = blockIdx.x; work < works; work += gridDim.x)
    {
        // the block's children: at most all of one parent
        const u32 child0 = next_first;
        const u32 last = min(next_end, ((child0 >> bits) + 1) << bits) - child0;        // parents without suffixes may lie between
        const bool more = work + gridDim.x < works;
        if(more) look_up(work + gridDim.x);
        const u32 first_digit = child0 & (children - 1);
        for(u32 d = tid; d <= last; d += BLOCK) coff[d] = __ldg(child_off + child0 + d);
        if(tid < 2) s_tied[tid] = 0;
        __syncthreads();
        u32 cur = 0;
        if(!MEDIUM && more)         // the next chunk's records on their way to L2: 16 to a line
        {
            const u64 at = u64(__ldg(child_off + next_first)) + tid * 16;
            if(at < list_cap) asm volatile("prefetch.global.L2 [%0];" :: "l"(rec + at));
        }

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
                if(e == cur)
                {
                    // a child that does not fit: left to the radix sort
                    if(tid == 0)
                    {
                        const u32 size = coff[cur + 1] - base;
                        if(!MEDIUM && size <= MEDIUM_CAP) over[over_cap - 1 - atomicAdd(&counts->medium, 1u)] = child0 + cur;
                        else
                        {
                            over[atomicAdd(&counts->oversize, 1u)] = child0 + cur;
                            atomicAdd(&counts->oversize_records, size);
                        }
                    }
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
                        if((tied >> i & 1u) && (pl[i] & PL_FIRST)) start[pl[i] & 8191u] = u16(atomicAdd(&s_tied[(pl[i] & PL_SMALL) ? 0 : 1], pl[i] >> 13 & 16383u));
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
        __syncthreads();            // a chunk may end in a child that was left or in an empty one: coff is still being read then
    }
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

bool wide_tiles(u64 n) { return n >= (u64(1) << 22); }         // small texts take small tiles, so that every SM gets one

}   // namespace

Prefix_Sort prefix_sort_plan(u64 n)
{
    Prefix_Sort ps;
    ps.n = n;
    int t = 0;                                          // children of at most 2048 suffixes on average
    while(t < MAX_B1 + MAX_B2 && (n >> t) > 2048) ++t;
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
    return align_up256(65536 * 4) * 2 + align_up256((size_t(1) << MAX_B1) * 4 + 4) * 5 + align_up256(all * 4) * 2 + align_up256((all + 1) * 4) + align_up256((ps.n / SHORT_CHUNK + (size_t(1) << MAX_B1) + 2) * 4) + 4096;
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
    t.chunk0 = cv.take<u32>((size_t(1) << MAX_B1) + 1);
    t.cnt2 = cv.take<u32>(all);
    t.child_off = cv.take<u32>(all + 1);
    t.over = cv.take<u32>(all);
    t.chunk_first = cv.take<u32>(ps.n / SHORT_CHUNK + (u64(1) << MAX_B1) + 2);
    return cv.ok;
}

namespace
{

// The code of the text's symbols; the counters of the first split and of the build are cleared on the way.
int launch_code(csa_ctx* ctx, const Prefix_Tables& t, const u16* T, const u64 n, Build_Counts* counts)
{
    // the code, from every symbol of a small text or a million of a large one
    static_assert(CODE_BLOCK == 1 << MAX_B1, "block 0 of make_code_kernel clears a counter of the first split per thread");
    if(n <= CODE_COUNT_MAX)
    {
        static std::atomic<bool> configured[64];
        CSA_TRY(shared_bytes(ctx, make_code_kernel<true>, CODE_SMEM, configured));
        make_code_kernel<true><<<65536 / CODE_WALKERS, CODE_BLOCK, CODE_SMEM, ctx->stream>>>(T, u32(n), nullptr, u32((u64(1) << 22) / n), t.code, t.cnt1, reinterpret_cast<u32*>(counts));
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
                     reinterpret_cast<u32*>(counts));
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

// The second split of `parents` buckets with n records in all (recA to recB).
int launch_second_split(csa_ctx* ctx, const Prefix_Tables& t, u32 parents, int b2, u64 n, const u64* recA, u64* recB)
{
    const unsigned tiles = unsigned(n / SPLIT_TILE + parents);
    const u32 children = 1u << b2;
    CSA_CUDA(ctx, cudaMemsetAsync(t.cnt2, 0, size_t(parents) * children * 4, ctx->stream));
    count_children_kernel<<<tiles, SPLIT_BLOCK, 0, ctx->stream>>>(recA, t.par_off, t.tile0, parents, b2, t.cnt2);
    CSA_LAUNCH_CHECK(ctx);
    child_offsets_kernel<<<parents, 1024, 0, ctx->stream>>>(t.cnt2, t.par_off, parents, children, t.child_off, t.chunk0, t.chunk_first);
    CSA_LAUNCH_CHECK(ctx);
    static std::atomic<bool> configured[64];
    CSA_TRY(shared_bytes(ctx, scatter_children_kernel, SPLIT_SMEM, configured));
    scatter_children_kernel<<<tiles, SPLIT_BLOCK, SPLIT_SMEM, ctx->stream>>>(recA, t.par_off, t.tile0, parents, b2, t.cnt2, recB);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

// The second launch takes the children of 4097 to 8192 suffixes; a short text, where a launch counts, goes to the larger blocks at once.
template <bool PACKED>
int launch_local_sort(csa_ctx* ctx, const Prefix_Tables& t, u32 parents, int b2, bool one_level, u64 n, const u64* rec, u32* sa, u8* sa40, u64* list, Build_Counts* counts)
{
    const u32 over_cap = parents << b2;
    const u32* const chunks = t.chunk0 + parents;
    if constexpr(PACKED)        // texts of one split are short
    {
        if(one_level)
        {
            static std::atomic<bool> configured[64];
            CSA_TRY(shared_bytes(ctx, local_sort_kernel<512, 16, 2, false, PACKED>, LOCAL_SMEM<512, 16>, configured));
            local_sort_kernel<512, 16, 2, false, PACKED><<<unsigned(n / SHORT_CHUNK + parents), 512, LOCAL_SMEM<512, 16>, ctx->stream>>>(rec, t.chunk_first, chunks, b2, t.child_off, sa, sa40, list, n, counts, t.over, over_cap);
            CSA_LAUNCH_CHECK(ctx);
            return CSA_OK;
        }
    }
    static std::atomic<bool> configured[2][64];
    CSA_TRY(shared_bytes(ctx, local_sort_kernel<512, 8, 3, false, PACKED>, LOCAL_SMEM<512, 8>, configured[0]));
    CSA_TRY(shared_bytes(ctx, local_sort_kernel<512, 16, 2, true, PACKED>, LOCAL_SMEM<512, 16>, configured[1]));
    local_sort_kernel<512, 8, 3, false, PACKED><<<unsigned(std::min<u64>(n / LOCAL_CHUNK + parents, 148 * 3 * 8)), 512, LOCAL_SMEM<512, 8>, ctx->stream>>>(rec, t.chunk_first, chunks, b2, t.child_off, sa, sa40, list, n, counts, t.over, over_cap);
    CSA_LAUNCH_CHECK(ctx);
    local_sort_kernel<512, 16, 2, true, PACKED><<<148 * 2, 512, LOCAL_SMEM<512, 16>, ctx->stream>>>(rec, t.chunk_first, chunks, b2, t.child_off, sa, sa40, list, n, counts, t.over, over_cap);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

}   // namespace

int launch_prefix_sort(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, u64* recA, u64* recB, u32* sa, u8* sa40, u32 p, Build_Counts* counts,
                       u64** list, u64** records, cudaEvent_t after_first_split)
{
    const u64 n = ps.n;
    CSA_TRY(launch_code(ctx, t, T, n, counts));
    const bool one_level = ps.b1 == 0;
    const int bits = one_level ? ps.b2 : ps.b1;
    if(bits > 0) CSA_TRY(launch_count_text(ctx, T, n, t.code, bits, t.cnt1));
    launch_early(parent_offsets_kernel, 1, 1024, 0, ctx->stream, t.cnt1, 1u << bits, u32(n), one_level ? 1 : 0, t.cur1, t.par_off, t.tile0, t.chunk0, t.child_off, t.chunk_first, p, counts);
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
        CSA_TRY(launch_second_split(ctx, t, ps.parents, ps.b2, n, recA, recB));
        rec = recB; other = recA;
    }
    CSA_TRY(sa ? launch_local_sort<false>(ctx, t, ps.parents, ps.b2, one_level, n, rec, sa, nullptr, other, counts)
               : launch_local_sort<true>(ctx, t, ps.parents, ps.b2, one_level, n, rec, nullptr, sa40, other, counts));
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
    CSA_TRY(launch_code(ctx, t, T, ps.n, counts));
    return launch_count_text(ctx, T, ps.n, t.code, ps.b1, t.cnt1);
}

int launch_prefix_sort_part(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, u32 first_bin, u32 bins, u64 size, u64* recA, u64* recB, u32* sa,
                            Build_Counts* counts)
{
    CSA_CUDA(ctx, cudaMemsetAsync(counts, 0, sizeof(Build_Counts), ctx->stream));
    parent_offsets_kernel<<<1, 1024, 0, ctx->stream>>>(t.cnt1 + first_bin, bins, u32(size), 0, t.cur1, t.par_off, t.tile0, t.chunk0, t.child_off, t.chunk_first, 1, counts);
    CSA_LAUNCH_CHECK(ctx);
    CSA_TRY(wide_tiles(ps.n) ? (launch_scatter_text<512, true>(ctx, T, ps.n, t.code, ps.b1, 0, first_bin, bins, t.cur1, recA))
                             : (launch_scatter_text<128, true>(ctx, T, ps.n, t.code, ps.b1, 0, first_bin, bins, t.cur1, recA)));
    CSA_TRY(launch_second_split(ctx, t, bins, ps.b2, size, recA, recB));
    CSA_TRY(launch_local_sort<false>(ctx, t, bins, ps.b2, false, size, recB, sa, nullptr, recA, counts));
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
