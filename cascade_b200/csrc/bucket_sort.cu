// The stable sort of csa_sort_pairs by its top bits first, for keys whose top bits are evenly spread: the records are split into buckets
// of about a thousand by the top 3 to 15 sorted bits with one or two of radix_sort.cu's digit passes (stable, low digit first), and every
// bucket is then finished inside one block. A record moves two or three times, where a pass per 8 bits moves it up to eight
// times (31.25 M 64-bit keys with 4-byte values, whole calls: 2.20 ms, this way 0.94 ms; 10^6: 217 us, 94 us; 1000, in one block: 140 us, 24 us). The buckets are counted
// exactly before anything moves, and keys for which the digit passes are the better way go through those: where a bucket fits no block, and where so few digits differ
// that most passes are skipped. (31.25 M records by digit passes alone and with the look at the keys before: all equal 97 and 99 us, 16 bits at the top 620 and 630, 20 at the bottom
// 864 and 876, one key in half of the places 2067 and 2089. By buckets after all, but inside them by digits as a key stands a hundred times: 1979 and 1727.)
// A list that fits one block at all is a single bucket and takes one launch.
#include "common.cuh"
#include "sort.cuh"

#include <algorithm>
#include <atomic>

namespace
{

// ---- the buckets' counts -----------------------------------------------------------------------------------------------------

constexpr int COUNT_BLOCK = 1024, COUNT_UNROLL = 4;

// Of more records than this every block looks at the same COUNT_BLOCK of them first, spread over the list (2 us): where those say that the keys are not
// for buckets, the rest is not counted. (31.25 M equal keys: 97 us by skipped digit passes alone, 178 with all of them counted first.)
constexpr u64 LOOKED_AT_FIRST = u64(1) << 21;

// Digits of 8 bits from begin_bit on in which keys differ: the digit passes that are not skipped. differ: bits in which any two keys do.
__device__ __forceinline__ int digits_that_differ(const u64 differ, const int begin_bit, const int end_bit)
{
    int digits = 0;
    for(int shift = begin_bit; shift < end_bit; shift += 8)
        digits += (differ >> shift & ((1ull << min(8, end_bit - shift)) - 1)) != 0;
    return digits;
}

// One read of the keys; a block counts in shared memory (32 bits a counter, at most 128 KB, as many blocks as SMs). Bound by the read.
// found->differ: bits in which keys differ; found->uneven: the counts are not complete, the keys go through the digit passes.
__global__ void __launch_bounds__(COUNT_BLOCK) bucket_counts_kernel(const u64* __restrict__ keys, const u64 n, const int begin_bit, const int end_bit, const int bits,
                                                                   const int least_digits, u32* __restrict__ counts, Bucket_Findings* __restrict__ found)
{
    let_next_in();
    extern __shared__ u32 cnt[];
    __shared__ u32 s_differ[2];
    const int shift = end_bit - bits;
    const u32 buckets = 1u << bits, mask = buckets - 1;
    for(u32 i = threadIdx.x; i < buckets; i += COUNT_BLOCK) cnt[i] = 0;
    if(threadIdx.x < 2) s_differ[threadIdx.x] = 0;
    const u64 k0 = keys[0];
    u64 differ = 0;
    auto block_differ = [&]()
    {
        const u32 lo = __reduce_or_sync(0xFFFFFFFFu, u32(differ)), hi = __reduce_or_sync(0xFFFFFFFFu, u32(differ >> 32));
        if(lane_id() == 0) { atomicOr(&s_differ[0], lo); atomicOr(&s_differ[1], hi); }
    };
    __syncthreads();
    if(n > LOOKED_AT_FIRST)
    {
        const u64 k = keys[u64(threadIdx.x) * (n / COUNT_BLOCK)];
        const u32 b = u32(k >> shift) & mask;
        differ = k ^ k0;
        block_differ();
        // several times what a bucket that fits a block may show here, so that keys whose buckets all fit are hardly ever refused
        const u32 most = 8 + u32(4 * BUCKET_MAX_RECORDS * COUNT_BLOCK / n);
        const bool heavy = __syncthreads_or(atomicAdd(&cnt[b], 1u) >= most);
        if(heavy || digits_that_differ(u64(s_differ[1]) << 32 | s_differ[0], begin_bit, end_bit) < least_digits)
        {
            if(blockIdx.x == 0 && threadIdx.x == 0) found->uneven = 1;
            return;
        }
        cnt[b] = 0;
        __syncthreads();
    }
    const u64 lead = (reinterpret_cast<uintptr_t>(keys) & 8) ? 1 : 0;           // a list may start on an odd 8-byte boundary
    const u64 pairs = (n - lead) >> 1;
    const ulonglong2* const k2 = reinterpret_cast<const ulonglong2*>(keys + lead);
    for(u64 i = u64(blockIdx.x) * (COUNT_BLOCK * COUNT_UNROLL) + threadIdx.x; i < pairs; i += u64(gridDim.x) * (COUNT_BLOCK * COUNT_UNROLL))
    {
        ulonglong2 k[COUNT_UNROLL];
        #pragma unroll
        for(int j = 0; j < COUNT_UNROLL; ++j) if(i + u64(j) * COUNT_BLOCK < pairs) k[j] = k2[i + u64(j) * COUNT_BLOCK];
        #pragma unroll
        for(int j = 0; j < COUNT_UNROLL; ++j)
            if(i + u64(j) * COUNT_BLOCK < pairs)
            {
                atomicAdd(&cnt[u32(k[j].x >> shift) & mask], 1u);
                atomicAdd(&cnt[u32(k[j].y >> shift) & mask], 1u);
                differ |= (k[j].x ^ k0) | (k[j].y ^ k0);
            }
    }
    if(blockIdx.x == 0 && threadIdx.x == 0)
    {
        if(lead) atomicAdd(&cnt[u32(k0 >> shift) & mask], 1u);
        if((n - lead) & 1) { atomicAdd(&cnt[u32(keys[n - 1] >> shift) & mask], 1u); differ |= keys[n - 1] ^ k0; }
    }
    block_differ();
    __syncthreads();
    for(u32 i = threadIdx.x; i < buckets; i += COUNT_BLOCK)
        if(const u32 c = cnt[i]) atomicAdd(&counts[i], c);
    if(threadIdx.x == 0) atomicOr(&found->differ, u64(s_differ[1]) << 32 | s_differ[0]);
}

__device__ __forceinline__ u32 warp_inclusive_sum(u32 v)
{
    #pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const u32 t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if(int(lane_id()) >= o) v += t;
    }
    return v;
}

// Exclusive sum over a block of up to 1024 threads; warp_tot: a word per warp. Ends with a barrier.
template <int BLOCK>
__device__ __forceinline__ u32 block_exclusive_sum(const u32 v, u32* warp_tot)
{
    const u32 inc = warp_inclusive_sum(v);
    if(lane_id() == 31) warp_tot[threadIdx.x >> 5] = inc;
    __syncthreads();
    const u32 t = lane_id() < BLOCK / 32 ? warp_tot[lane_id()] : 0;
    const u32 pre = __shfl_sync(0xFFFFFFFFu, warp_inclusive_sum(t) - t, threadIdx.x >> 5);
    __syncthreads();
    return pre + inc - v;
}

// One block: the counts become the buckets' starts, in place (starts[buckets] = n); the digit offsets of the one or two passes by which
// the records get there (low digit first: low_bits of them, which may be 0, then the top bits); and the verdict: found->uneven where a bucket does not fit a
// block or fewer than least_digits digits differ. verdict (pinned host memory): the largest bucket, 0 for uneven keys.
__global__ void __launch_bounds__(1024) bucket_plan_kernel(u32* __restrict__ counts, const u32 n, const int begin_bit, const int end_bit, const int bits, const int low_bits,
                                                          const int least_digits, u64* __restrict__ low_base, u64* __restrict__ high_base, Bucket_Findings* __restrict__ found,
                                                          u64* __restrict__ verdict)
{
    let_next_in();
    wait_for_previous();
    if(found->uneven) { if(threadIdx.x == 0) *verdict = 0; return; }
    __shared__ u32 warp_tot[32];
    __shared__ u32 low[256];
    __shared__ u32 most;
    const u32 t = threadIdx.x, buckets = 1u << bits, lane = lane_id(), warp = t >> 5;
    if(t < 256) low[t] = 0;
    if(t == 0) most = 0;
    __syncthreads();
    if(low_bits)        // thread t: the buckets t + k * 1024, whose low digits are the same
    {
        u32 s = 0;
        #pragma unroll 8
        for(u32 i = t; i < buckets; i += 1024) s += counts[i];
        if(s) atomicAdd(&low[t & ((1u << low_bits) - 1)], s);
    }
    u32 big = 0;
    if(buckets <= 1024)
    {
        const u32 c = t < buckets ? counts[t] : 0;
        big = c;
        const u32 at = block_exclusive_sum<1024>(c, warp_tot);
        if(t < buckets) { counts[t] = at; if((t & ((1u << low_bits) - 1)) == 0) high_base[t >> low_bits] = at; }
    }
    else
    {
        // a warp sums buckets / 32 counts side by side, 128 at a time (a thread its 32 one by one: 62 us for 2^15 buckets, this way 10 us); there are
        // two low bits or more, so every fourth bucket may start a high digit's run
        const u32 span = buckets / 32;
        constexpr int ROUNDS = (1 << BUCKET_MAX_BITS) / 32 / 128;
        uint4 c[ROUNDS];
        u32 at[ROUNDS], run = 0;
        #pragma unroll
        for(int k = 0; k < ROUNDS; ++k)
        {
            const u32 i = k * 128 + lane * 4;
            c[k] = i < span ? *reinterpret_cast<const uint4*>(counts + warp * span + i) : make_uint4(0, 0, 0, 0);
        }
        #pragma unroll
        for(int k = 0; k < ROUNDS; ++k)
        {
            const u32 sum = c[k].x + c[k].y + c[k].z + c[k].w, inc = warp_inclusive_sum(sum);
            big = max(big, max(max(c[k].x, c[k].y), max(c[k].z, c[k].w)));
            at[k] = run + inc - sum;
            run += __shfl_sync(0xFFFFFFFFu, inc, 31);
        }
        if(lane == 31) warp_tot[warp] = run;
        __syncthreads();
        const u32 tot = warp_tot[lane];
        const u32 before = __shfl_sync(0xFFFFFFFFu, warp_inclusive_sum(tot) - tot, warp);
        __syncthreads();
        #pragma unroll
        for(int k = 0; k < ROUNDS; ++k)
        {
            const u32 i = k * 128 + lane * 4;
            if(i >= span) continue;
            const u32 b = warp * span + i, x = before + at[k], y = x + c[k].x, z = y + c[k].y, w = z + c[k].z;
            *reinterpret_cast<uint4*>(counts + b) = make_uint4(x, y, z, w);
            if((b & ((1u << low_bits) - 1)) == 0) high_base[b >> low_bits] = x;
        }
    }
    big = __reduce_max_sync(0xFFFFFFFFu, big);
    if(lane == 0) atomicMax(&most, big);
    __syncthreads();
    const u32 at = block_exclusive_sum<1024>(t < 256 ? low[t] : 0, warp_tot);
    if(low_bits && t < (1u << low_bits)) low_base[t] = at;
    if(t == 0)
    {
        counts[buckets] = n;
        const bool even = most <= BUCKET_MAX_RECORDS && digits_that_differ(found->differ, begin_bit, end_bit) >= least_digits;
        found->uneven = even ? 0 : 1;
        *verdict = even ? most : 0;
    }
}

// ---- a bucket inside one block -------------------------------------------------------------------------------------------------

constexpr int BUCKET_ITEMS = 8;
template <int BLOCK> constexpr u32 BUCKET_CAP = BLOCK * BUCKET_ITEMS;
constexpr u32 LONG_BIN = 24;       // a bin with more records is not ordered by comparing all with all
// the staged keys; then the bins and the places before, and where those were, the values
template <int BLOCK, typename V> constexpr size_t BUCKET_SMEM = size_t(BUCKET_CAP<BLOCK>) * 8 + (sizeof(V) == 8 ? size_t(BUCKET_CAP<BLOCK>) * 8 : size_t(BUCKET_CAP<BLOCK>) * 4 + 32);

// Sorts every bucket [starts[b], starts[b + 1]) (starts == nullptr: one bucket, [0, n)) by the bits `compared` of its keys, of which
// the highest is bit top - 1, stably, from the `in` to the `out` arrays. There are as many bins as records (up to a factor of 2): a record's
// bin is its next key bits, its place in the bin is what a shared-memory atomic hands out, and inside the bin it counts the keys before its own, equal ones
// by the places they came from. So the order is the stable one whatever order the atomics took. A record stays with its thread until its place is known; keys
// and values then go out by way of shared memory, side by side.
// A bin of more than LONG_BIN records sends the bucket through stable passes by digits instead, as many as its keys differ in (8192 equal keys in one block: 120 us by a sorting
// network, 30 this way). Even keys have no such bin. Thirty records a key, 31.25 M records, in a row and far apart: with bins of up to 40 compared 1.49 and 2.20 ms, of up to 24
// 1.71 and 1.79; by digit passes alone 2.03 and 2.12. What bounds it is the issue of instructions and barriers between
// dependent steps: blocks are as small as the largest bucket allows, with 8 records a thread. (31.25 M records, 16 a thread and the values
// gathered when the places were known: 454 us, this way 389 us.)
template <int BLOCK, int ITEMS, typename V>
__device__ __forceinline__ void sort_bucket(unsigned char* const smem_raw, const u64* __restrict__ keys_in, u64* __restrict__ keys_out, const V* __restrict__ vals_in, V* __restrict__ vals_out,
                                            const u32 base, const u32 m, const u64 compared, const int top, const int begin)
{
    constexpr u32 CAP = BLOCK * ITEMS;
    u64* const stage = reinterpret_cast<u64*>(smem_raw);            // [CAP]
    u32* const bin = reinterpret_cast<u32*>(stage + CAP);           // [CAP / 2 + 8]: two 16-bit counters a word, then the bins' starts
    u16* const start = reinterpret_cast<u16*>(bin);
    u16* const from = reinterpret_cast<u16*>(bin + CAP / 2 + 8);    // [CAP]: the record's place in the bucket before
    V* const vals = reinterpret_cast<V*>(stage + CAP);              // [CAP], once the bins are no longer needed
    __shared__ u32 warp_tot[BLOCK / 32], s_differ[2];
    static_assert(BLOCK / 32 * 256 <= CAP && BLOCK >= 256 && CAP <= 8192, "the warps' counts lie where the bins do; places take 13 bits");
    const u32 tid = threadIdx.x;
    if(m == 0 || m > CAP) return;       // the host has seen to it that all fit
    keys_in += base; keys_out += base;
    if(vals_in != nullptr) { vals_in += base; vals_out += base; }

    const int bin_bits = min(min(32 - __clz(m - 1 | 1u), 31 - __clz(CAP)), top - begin);     // bins: a power of two, at most CAP
    const u32 bins = 1u << bin_bits;
    const int bin_shift = top - bin_bits;
    const u32 bin_mask = bins - 1;
    for(u32 i = tid; i < (bins / 2 + 8) / 4; i += BLOCK) reinterpret_cast<uint4*>(bin)[i] = make_uint4(0, 0, 0, 0);
    u64 r[ITEMS];
    u32 pl[ITEMS];                      // place in the bin, later in the bucket
    #pragma unroll
    for(int i = 0; i < ITEMS; ++i)
    {
        if(i * BLOCK >= m) break;
        const u32 j = tid + i * BLOCK;
        if(j < m) r[i] = keys_in[j];
    }
    __syncthreads();
    auto bin_of = [&](const u64 key) { return u32(key >> bin_shift) & bin_mask; };
    #pragma unroll
    for(int i = 0; i < ITEMS; ++i)
    {
        if(i * BLOCK >= m) break;
        if(tid + i * BLOCK < m)
        {
            const u32 b = bin_of(r[i]);
            const u32 old = atomicAdd(&bin[b >> 1], (b & 1) ? 0x10000u : 1u);
            pl[i] = (b & 1) ? old >> 16 : old & 0xFFFFu;
        }
    }
    __syncthreads();
    // exclusive sums of the bins' counts, in place; start[bins] = m
    u32 longest = 0;
    {
        constexpr int WORDS = CAP / 2 / BLOCK;
        u32 c[WORDS], sum = 0;
        const bool any = tid * WORDS * 2 <= bins;       // the words up to a multiple of WORDS were cleared
        if(any)
        {
            #pragma unroll
            for(int k = 0; k < WORDS; ++k) c[k] = bin[tid * WORDS + k];
            u32 both = 0;
            #pragma unroll
            for(int k = 0; k < WORDS; ++k) { both += c[k]; longest = __vmaxu2(longest, c[k]); }
            sum = (both & 0xFFFFu) + (both >> 16);
        }
        const u32 inc = warp_inclusive_sum(sum);
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
                bin[tid * WORDS + k] = a;
            }
        }
        if(bins == CAP && tid == 0) start[CAP] = u16(m);            // behind the threads' words
    }
    if(__syncthreads_or(max(longest & 0xFFFFu, longest >> 16) > LONG_BIN))
    {
        // Many records in one bin: stable passes by 8 of the bits in which the bucket's keys differ, low ones first. A warp takes up to 256 records in a row and
        // numbers those of a digit itself; the sums over the warps' counts give the places.
        const u32 rounds = (m + BLOCK - 1) / BLOCK;         // 32 records a warp in each
        u16 (*const count)[256] = reinterpret_cast<u16 (*)[256]>(bin);
        const u32 warp = tid >> 5, lane = lane_id();
        if(tid < 2) s_differ[tid] = 0;
        #pragma unroll
        for(int i = 0; i < ITEMS; ++i)
        {
            const u32 j = tid + i * BLOCK;
            if(j >= m) break;
            stage[j] = r[i];
            from[j] = u16(j);
        }
        __syncthreads();
        {
            u64 differ = 0;
            const u64 k0 = stage[0];
            #pragma unroll
            for(int i = 0; i < ITEMS; ++i) if(tid + i * BLOCK < m) differ |= r[i] ^ k0;
            differ &= compared;
            const u32 lo = __reduce_or_sync(0xFFFFFFFFu, u32(differ)), hi = __reduce_or_sync(0xFFFFFFFFu, u32(differ >> 32));
            if(lane == 0) { atomicOr(&s_differ[0], lo); atomicOr(&s_differ[1], hi); }
        }
        __syncthreads();
        for(u64 rest = u64(s_differ[1]) << 32 | s_differ[0]; rest; )
        {
            const int shift = __ffsll(rest) - 1;
            rest = shift + 8 >= 64 ? 0 : rest & (~0ull << (shift + 8));
            reinterpret_cast<uint4*>(count[warp])[lane] = make_uint4(0, 0, 0, 0);
            __syncwarp();
            auto digit_of = [&](const u64 key) { return u32((key & compared) >> shift) & 255u; };
            const u32 first = warp * (32 * rounds) + lane;
            #pragma unroll
            for(int i = 0; i < ITEMS; ++i)
                if(i < rounds && first + i * 32 < m) { r[i] = stage[first + i * 32]; pl[i] = from[first + i * 32]; }
            #pragma unroll
            for(int i = 0; i < ITEMS; ++i)
            {
                if(i >= rounds) break;
                const bool there = first + i * 32 < m;
                const u32 d = there ? digit_of(r[i]) : 256u, same = __match_any_sync(0xFFFFFFFFu, d);
                const u32 before = there ? count[warp][d] : 0u;
                __syncwarp();
                if(there)
                {
                    pl[i] |= (before + __popc(same & lanemask_lt())) << 16;
                    if(lane == u32(__ffs(same)) - 1) count[warp][d] = u16(before + __popc(same));
                }
                __syncwarp();
            }
            __syncthreads();
            u32 sum = 0;
            if(tid < 256)
                for(u32 w = 0; w < BLOCK / 32; ++w) sum += count[w][tid];
            u32 run = block_exclusive_sum<BLOCK>(sum, warp_tot);
            if(tid < 256)
                for(u32 w = 0; w < BLOCK / 32; ++w) { const u32 c = count[w][tid]; count[w][tid] = u16(run); run += c; }
            __syncthreads();
            #pragma unroll
            for(int i = 0; i < ITEMS; ++i)
                if(i < rounds && first + i * 32 < m)
                {
                    const u32 at = count[warp][digit_of(r[i])] + (pl[i] >> 16);
                    stage[at] = r[i];
                    from[at] = u16(pl[i]);
                }
            __syncthreads();
        }
        for(u32 j = tid; j < m; j += BLOCK)
        {
            keys_out[j] = stage[j];
            if(vals_in != nullptr) vals_out[j] = vals_in[from[j]];
        }
        return;
    }
    #pragma unroll
    for(int i = 0; i < ITEMS; ++i)
    {
        if(i * BLOCK >= m) break;
        const u32 j = tid + i * BLOCK;
        if(j < m)
        {
            const u32 at = start[bin_of(r[i])] + pl[i];
            stage[at] = r[i] & compared;
            from[at] = u16(j);
        }
    }
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < ITEMS; ++i)
    {
        if(i * BLOCK >= m) break;
        const u32 f = tid + i * BLOCK;
        if(f < m)
        {
            const u64 mine = r[i] & compared;
            const u32 b = bin_of(r[i]), s = start[b], e = start[b + 1];
            u32 less = 0, upto = 0;
            #pragma unroll
            for(u32 k = 0; k < 3; ++k)          // most bins hold no more: three reads in flight
                if(s + k < e) { const u64 o = stage[s + k]; less += o < mine; upto += o <= mine; }
            for(u32 k = s + 3; k < e; ++k) { const u64 o = stage[k]; less += o < mine; upto += o <= mine; }
            u32 place = s + less;
            if(upto - less > 1)
                for(u32 k = s; k < e; ++k) place += stage[k] == mine && from[k] < f;
            pl[i] = place;
        }
    }
    __syncthreads();        // the bins and the keys in them have been read
    #pragma unroll
    for(int i = 0; i < ITEMS; ++i)
    {
        if(i * BLOCK >= m) break;
        const u32 j = tid + i * BLOCK;
        if(j < m)
        {
            stage[pl[i]] = r[i];
            if(vals_in != nullptr) vals[pl[i]] = vals_in[j];
        }
    }
    __syncthreads();
    #pragma unroll
    for(int i = 0; i < ITEMS; ++i)
    {
        const u32 j = tid + i * BLOCK;
        if(j >= m) break;
        keys_out[j] = stage[j];
        if(vals_in != nullptr) vals_out[j] = vals[j];
    }
}

template <int BLOCK, int BLOCKS, typename V>
__global__ void __launch_bounds__(BLOCK, BLOCKS) bucket_sort_kernel(const u64* __restrict__ keys_in, u64* __restrict__ keys_out, const V* __restrict__ vals_in, V* __restrict__ vals_out,
                                                                   const u32* __restrict__ starts, const u32 n, const u64 compared, const int top, const int begin)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const u32 base = starts ? starts[blockIdx.x] : 0, m = (starts ? starts[blockIdx.x + 1] : n) - base;
    sort_bucket<BLOCK, BUCKET_ITEMS, V>(smem_raw, keys_in, keys_out, vals_in, vals_out, base, m, compared, top, begin);
}

// Apart, so that the kernel below keeps its registers.
template <int BLOCK, int ITEMS, typename V>
__device__ __noinline__ void sort_bucket_apart(unsigned char* const smem_raw, const u64* __restrict__ keys_in, u64* __restrict__ keys_out, const V* __restrict__ vals_in, V* __restrict__ vals_out,
                                               const u32 base, const u32 m, const u64 compared, const int top, const int begin)
{
    sort_bucket<BLOCK, ITEMS, V>(smem_raw, keys_in, keys_out, vals_in, vals_out, base, m, compared, top, begin);
}

// ---- a bucket inside one block, evenly spread keys -----------------------------------------------------------------------------------------

constexpr int ORDER_BLOCK = 256;
// words of the records and their bins; then their keys and values as they came
template <int ITEMS> constexpr u32 ORDER_CAP = ORDER_BLOCK * ITEMS;
template <int ITEMS> constexpr u32 ORDER_MOST = ORDER_CAP<ITEMS> - 4;
template <int ITEMS, typename V> constexpr size_t ORDER_SMEM = size_t(ORDER_CAP<ITEMS>) * (4 + 2 + 8 + sizeof(V)) + 80;
constexpr int FROM_BITS = 12, WORD_BITS = 32 - FROM_BITS;       // a word: the first bits of a key that the buckets do not tell, and the record's place in the bucket before
constexpr u32 MOST_CROWDED = 64;
// Four counts of five bits a word, later where the word's records begin (12 bits) and, in the fields, where those of each bin do.
constexpr u32 each_bin(const u32 v) { return v | v << 5 | v << 10 | v << 15; }
constexpr u32 SUMS = each_bin(1) << 5, SUMS_BEFORE = each_bin(31) & ~31u, SUM_OF_ALL = 31u << 20;
constexpr u32 TO_EIGHT = each_bin(3), EIGHT_UP = each_bin(24), FULL_BIN = each_bin(16);

__device__ __forceinline__ void order(u32& a, u32& b) { const u32 t = min(a, b); b = max(a, b); a = t; }
__device__ __forceinline__ void order(u32& a, u32& b, u32& c) { order(a, b); order(b, c); order(a, b); }

// As the resident build's local sort: records are counted in two bins each by interpolation of their words, the words go to shared memory in the order of the bins, and a thread orders
// the words of four slots with those of the three slots before and behind by min and max: bins of up to four records lie inside the window of every slot of theirs, the few of up to 15 are
// ordered by a warp. A word ends in the record's place in the bucket before, so equal keys stay in their order; where a word does not hold all compared bits, records of the same first bits
// are told apart by their whole keys. Keys and values are read from shared memory by that place and go out as 16-byte stores.
// A bucket with a bin of 16 or more is sorted as above; where one in eight is, the others are not tried in this way.
// Bound by the issue of instructions (159 for 32 records, 48 % of the cycles) and the chain of a single bucket in a block: 31.25 M records of 64-bit keys and 4-byte values in buckets of 1907, 296 us where
// bucket_sort_kernel takes 378; whole calls 1123 -> 1034 us, by 32 bits 972 -> 834.
template <int ITEMS, int BLOCKS, typename V>
__global__ void __launch_bounds__(ORDER_BLOCK, BLOCKS) order_buckets_kernel(const u64* __restrict__ keys_in, u64* __restrict__ keys_out, const V* __restrict__ vals_in, V* __restrict__ vals_out,
                                                                            const u32* __restrict__ starts, Bucket_Findings* __restrict__ found, const u64 compared, const int top, const int begin)
{
    constexpr u32 BLOCK = ORDER_BLOCK, CAP = ORDER_CAP<ITEMS>, WARPS = BLOCK / 32, WORDS = CAP / 2 / BLOCK, CROWD_WORDS = CAP / 32 + 4;
    static_assert(CAP <= 1u << FROM_BITS && CROWD_WORDS <= BLOCK && WORDS * 2 * BLOCK == CAP, "places take 12 bits");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u64* const key = reinterpret_cast<u64*>(smem_raw);                  // [CAP]
    V* const val = reinterpret_cast<V*>(key + CAP);                     // [CAP]
    u32* const words = reinterpret_cast<u32*>(val + CAP) + 4;           // [CAP + 16] in the order of the bins; four before it
    u32* const bin = words + CAP + 16;                                  // [CAP / 2]
    __shared__ u32 warp_tot[WARPS], crowd[CROWD_WORDS], crowded[MOST_CROWDED], s_crowded, s_fall;
    __shared__ u32 s_untried;       // apart from s_fall, which a thread that is ahead sets while another still asks whether the bucket is tried
    const u32 tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const u32 base = starts[blockIdx.x], m = starts[blockIdx.x + 1] - base;
    if(m == 0) return;
    const u32 full = __shfl_sync(0xFFFFFFFFu, m / BLOCK, 0), rest = m % BLOCK, shift = base & 3u, end = shift + m, whole = base - shift;
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
    u64 r[ITEMS];
    V v[ITEMS];
    for_each([&](const u32 i, const u32 j) { r[i] = keys_in[base + j]; if(vals_in != nullptr) v[i] = vals_in[base + j]; });
    #pragma unroll
    for(u32 w = 0; w < WORDS; ++w) bin[tid + w * BLOCK] = 0;
    if(tid < CROWD_WORDS) crowd[tid] = 0;
    if(tid < 4) words[int(tid) - 4] = 0;
    if(tid == 0) { s_crowded = 0; s_fall = 0; s_untried = found->left > blockIdx.x / 8 + 64; }
    u32 k[ITEMS];
    for_each([&](const u32 i, const u32 j)
    {
        key[j] = r[i];
        if(vals_in != nullptr) val[j] = v[i];
        k[i] = u32(((r[i] & compared) << (64 - top)) >> 32) & ~((1u << FROM_BITS) - 1);
    });
    __syncthreads();
    if(s_untried)
    {
        sort_bucket_apart<ORDER_BLOCK, ITEMS, V>(smem_raw, keys_in, keys_out, vals_in, vals_out, base, m, compared, top, begin);
        return;
    }
    u32 seen = 0, number[(ITEMS + 7) / 8] = {};
    for_each([&](const u32 i, const u32)
    {
        const u32 b = __umulhi(k[i], 2 * m), old = atomicAdd(bin + (b >> 2), 1u << (5 * (b & 3u)));
        seen |= old;
        number[i / 8] |= (old >> (5 * (b & 3u)) & 15u) << (4 * (i % 8));
    });
    if(seen & FULL_BIN) s_fall = 1;
    __syncthreads();
    const bool any = 2 * WORDS * tid < m, busy = 64 * WORDS * warp < m;
    u32 c[WORDS], sum = 0, inc = 0, many = 0;
    if(busy)
    {
        #pragma unroll
        for(u32 w = 0; w < WORDS; ++w)
        {
            c[w] = any ? bin[WORDS * tid + w] : 0u;
            many |= (c[w] + TO_EIGHT) & EIGHT_UP;
            sum += c[w] * SUMS & SUM_OF_ALL;
        }
        inc = warp_inclusive_sum(sum);
    }
    if(lane == 31) warp_tot[warp] = inc;
    __syncthreads();
    if(busy)
    {
        u32 run = (shift << 20) + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? warp_tot[lane] : 0u) + inc - sum;
        if(any)
        {
            #pragma unroll
            for(u32 w = 0; w < WORDS; ++w) { bin[WORDS * tid + w] = (c[w] * SUMS & SUMS_BEFORE) | run; run += c[w] * SUMS & SUM_OF_ALL; }
        }
        if(many)
        {
            #pragma unroll
            for(u32 w = 0; w < WORDS; ++w)
                #pragma unroll 1
                for(u32 f = (c[w] + TO_EIGHT) & EIGHT_UP; f;)
                {
                    const u32 bit = (__ffs(f) - 1) / 5 * 5, size = c[w] >> bit & 31u, x = bin[WORDS * tid + w];
                    const u32 at = (x >> 20) + (x >> bit & 31u), o = atomicAdd(&s_crowded, 1u);
                    f &= ~(31u << bit);
                    if(o < MOST_CROWDED) crowded[o] = at | size << 16;
                    const u64 marks = u64((1u << size) - 1) << (at & 31u);
                    if((at >> 5) + 1 < CROWD_WORDS)
                    {
                        atomicOr(&crowd[at >> 5], u32(marks));
                        if(marks >> 32) atomicOr(&crowd[(at >> 5) + 1], u32(marks >> 32));
                    }
                    u32 all = 0;
                    for(int b = 0; b < 4; ++b) all += c[w] >> (5 * b) & 31u;
                    if(o >= MOST_CROWDED || (c[w] & FULL_BIN) || all > 31) s_fall = 1;
                }
        }
    }
    __syncthreads();
    if(s_fall)
    {
        if(tid == 0) atomicAdd(&found->left, 1u);
        sort_bucket_apart<ORDER_BLOCK, ITEMS, V>(smem_raw, keys_in, keys_out, vals_in, vals_out, base, m, compared, top, begin);
        return;
    }
    for_each([&](const u32 i, const u32 j)
    {
        const u32 b = __umulhi(k[i], 2 * m), x = bin[b >> 2], slot = (x >> 20) + (x >> (5 * (b & 3u)) & 31u) + (number[i / 8] >> (4 * (i % 8)) & 15u);
        words[slot] = k[i] | j;
    });
    if(tid < shift) words[tid] = 0;                     // no word is below, or above those behind
    if(tid < 8) words[end + tid] = 0xFFFFFFFFu;
    __syncthreads();
    constexpr u32 FROM = (1u << FROM_BITS) - 1;
    const bool told = top - begin <= WORD_BITS;         // a word holds all of a key that is compared
    const bool aligned = ((reinterpret_cast<uintptr_t>(keys_out) | reinterpret_cast<uintptr_t>(vals_out)) & 15) == 0;
    // The record of a group of the same first bits that comes at place `rank` of it; the group lies inside the slots [first, stop).
    auto whole_less = [&](const u32 a, const u32 b) { const u64 x = key[a & FROM] & compared, y = key[b & FROM] & compared; return x < y || (x == y && a < b); };
    const u32 crowds = s_crowded;
    #pragma unroll 1
    for(u32 q0 = warp * 32; 4 * q0 < end; q0 += BLOCK)
    {
        const u32 q = q0 + lane;
        const uint4* const K = reinterpret_cast<const uint4*>(words - 4) + q;
        const uint4 L = K[0], O = K[1], R = K[2];
        u32 a0 = L.y, a1 = L.z, a2 = L.w, x0 = O.x, x1 = O.y, x2 = O.z, x3 = O.w, r0 = R.x, r1 = R.y, r2 = R.z;
        order(x0, x1); order(x2, x3); order(x0, x2); order(x1, x3); order(x1, x2);
        order(a0, a1, a2);
        order(r0, r1, r2);
        const u32 before = max(max(min(a0, x2), min(a1, x1)), min(a2, x0));
        x2 = max(a0, x2); x1 = max(a1, x1); x0 = max(a2, x0);
        order(x0, x1, x2);
        const u32 behind = min(min(max(x1, r2), max(x2, r1)), max(x3, r0));
        x1 = min(x1, r2); x2 = min(x2, r1); x3 = min(x3, r0);
        order(x1, x2, x3);
        u32 x[4] = {x0, x1, x2, x3};
        u32 wanted = 4 * q < end ? 15u : 0u;
        if(4 * q < shift) wanted = 15u << shift & 15u;
        if(4 * q + 4 > end && wanted) wanted &= 15u >> (4 * q + 4 - end);
        if(crowds) wanted &= ~(crowd[q >> 3] >> (4 * (q & 7u)));
        if(!told && min(min(min(before ^ x0, x0 ^ x1), min(x1 ^ x2, x2 ^ x3)), x3 ^ behind) <= FROM)
        {
            #pragma unroll
            for(u32 i = 0; i < 4; ++i)
            {
                if(!(wanted >> i & 1u)) continue;
                const u32 mine = x[i], first = max(4 * q + i, shift + 3) - 3, stop = min(4 * q + i + 4, end);
                u32 rank = 0, group = 0;
                #pragma unroll 1
                for(u32 s = first; s < stop; ++s)
                    if((words[s] ^ mine) <= FROM) { ++group; rank += words[s] < mine; }
                if(group <= 1) continue;
                #pragma unroll 1
                for(u32 s = first; s < stop; ++s)
                {
                    if((words[s] ^ mine) > FROM) continue;
                    u32 less = 0;
                    #pragma unroll 1
                    for(u32 o = first; o < stop; ++o)
                        if((words[o] ^ mine) <= FROM && whole_less(words[o], words[s])) ++less;
                    if(less == rank) x[i] = words[s];
                }
            }
        }
        const u64 to = u64(whole) + 4 * q;
        if(aligned && wanted == 15u)
        {
            reinterpret_cast<ulonglong2*>(keys_out + to)[0] = make_ulonglong2(key[x[0] & FROM], key[x[1] & FROM]);
            reinterpret_cast<ulonglong2*>(keys_out + to)[1] = make_ulonglong2(key[x[2] & FROM], key[x[3] & FROM]);
            if(vals_in != nullptr)
            {
                if constexpr(sizeof(V) == 4) *reinterpret_cast<uint4*>(vals_out + to) = make_uint4(val[x[0] & FROM], val[x[1] & FROM], val[x[2] & FROM], val[x[3] & FROM]);
                else
                {
                    reinterpret_cast<ulonglong2*>(vals_out + to)[0] = make_ulonglong2(val[x[0] & FROM], val[x[1] & FROM]);
                    reinterpret_cast<ulonglong2*>(vals_out + to)[1] = make_ulonglong2(val[x[2] & FROM], val[x[3] & FROM]);
                }
            }
        }
        else
            #pragma unroll
            for(u32 i = 0; i < 4; ++i)
                if(wanted >> i & 1u)
                {
                    keys_out[to + i] = key[x[i] & FROM];
                    if(vals_in != nullptr) vals_out[to + i] = val[x[i] & FROM];
                }
    }
    #pragma unroll 1
    for(u32 o = WARPS - 1 - warp; o < crowds; o += WARPS)
    {
        const u32 s = crowded[o] & 0xFFFFu, size = crowded[o] >> 16;
        const u32 mine = words[s + min(lane, size - 1)];
        u32 less = 0;
        #pragma unroll 1
        for(u32 j = 0; j < size; ++j) less += whole_less(words[s + j], mine);
        if(lane < size)
        {
            keys_out[u64(whole) + s + less] = key[mine & FROM];
            if(vals_in != nullptr) vals_out[u64(whole) + s + less] = val[mine & FROM];
        }
    }
}

template <int ITEMS, int BLOCKS, typename V>
int launch_order(csa_ctx* ctx, const u64* kin, u64* kout, const V* vin, V* vout, const u32* starts, u32 buckets, Bucket_Findings* found, u64 compared, int top, int begin)
{
    static std::atomic<bool> configured[64];
    static_assert(ORDER_SMEM<ITEMS, V> >= size_t(ORDER_CAP<ITEMS>) * 8 + (sizeof(V) == 8 ? size_t(ORDER_CAP<ITEMS>) * 8 : size_t(ORDER_CAP<ITEMS>) * 4 + 32), "room for sort_bucket");
    if(!configured[ctx->device & 63])
    {
        CSA_CUDA(ctx, cudaFuncSetAttribute(order_buckets_kernel<ITEMS, BLOCKS, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(ORDER_SMEM<ITEMS, V>)));
        configured[ctx->device & 63] = true;
    }
    order_buckets_kernel<ITEMS, BLOCKS, V><<<buckets, ORDER_BLOCK, ORDER_SMEM<ITEMS, V>, ctx->stream>>>(kin, kout, vin, vout, starts, found, compared, top, begin);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

template <int BLOCK, int BLOCKS, typename V>
int launch_buckets(csa_ctx* ctx, const u64* kin, u64* kout, const V* vin, V* vout, const u32* starts, u32 buckets, u64 n, u64 compared, int top, int begin)
{
    static std::atomic<bool> configured[64];
    if(!configured[ctx->device & 63])
    {
        CSA_CUDA(ctx, cudaFuncSetAttribute(bucket_sort_kernel<BLOCK, BLOCKS, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(BUCKET_SMEM<BLOCK, V>)));
        configured[ctx->device & 63] = true;
    }
    bucket_sort_kernel<BLOCK, BLOCKS, V><<<buckets, BLOCK, BUCKET_SMEM<BLOCK, V>, ctx->stream>>>(kin, kout, vin, vout, starts, u32(n), compared, top, begin);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

// 31.25 M records: see the kernel; 4 and 1 M the same either way; 1e5 with few bits that differ 64 us by bucket_sort_kernel, 76 by order_buckets_kernel, which leaves such buckets after a try.
constexpr u64 ORDER_MIN = u64(1) << 22;
// The largest of its blocks only where a word holds all that is compared and the buckets are as large as those of random keys (seven standard deviations above their mean): 5.5e7 records by 32 bits 1647 and 1340 us,
// but by 64 bits, where the registers do not do, 1584 and 1635 (two blocks an SM 1760), and of keys that stand eight or 64 times, whose buckets are left after a try, by 32 bits and with 8-byte values 2520 and 2810.

template <typename V>
int launch_buckets_of(csa_ctx* ctx, const u64* kin, u64* kout, const V* vin, V* vout, const u32* starts, u32 buckets, u64 n, u64 largest, Bucket_Findings* found, int begin, int top)
{
    const u64 compared = (top >= 64 ? ~0ull : (1ull << top) - 1) & (~0ull << begin);
    if(n >= ORDER_MIN)
    {
        if(largest <= ORDER_MOST<8>) return launch_order<8, 5, V>(ctx, kin, kout, vin, vout, starts, buckets, found, compared, top, begin);
        if(largest <= ORDER_MOST<10>) return launch_order<10, 4, V>(ctx, kin, kout, vin, vout, starts, buckets, found, compared, top, begin);
        const u64 mean = n / buckets, over = largest - mean;
        if(largest <= ORDER_MOST<16> && top - begin <= WORD_BITS && over * over <= 49 * mean) return launch_order<16, sizeof(V) == 4 ? 3 : 2, V>(ctx, kin, kout, vin, vout, starts, buckets, found, compared, top, begin);
    }
    if(largest <= BUCKET_CAP<256>) return launch_buckets<256, 6, V>(ctx, kin, kout, vin, vout, starts, buckets, n, compared, top, begin);
    if(largest <= BUCKET_CAP<512>) return launch_buckets<512, 3, V>(ctx, kin, kout, vin, vout, starts, buckets, n, compared, top, begin);
    if(largest <= BUCKET_CAP<1024>) return launch_buckets<1024, 1, V>(ctx, kin, kout, vin, vout, starts, buckets, n, compared, top, begin);
    return csa_fail(ctx, CSA_E_DEVICE, "bucket sort: a bucket does not fit a block");
}

static_assert(BUCKET_CAP<1024> == BUCKET_MAX_RECORDS, "");

}   // namespace

int bucket_sort_bits(u64 n)
{
    int t = 0;
    while(t < BUCKET_MAX_BITS && (n >> t) > 1024) ++t;
    return t == 9 ? 8 : t;          // 9 bits would be a second pass
}

int launch_bucket_plan(csa_ctx* ctx, const u64* keys, u64 n, int begin_bit, int end_bit, int bits, int low_bits, int least_digits, u32* starts, u64* low_base, u64* high_base,
                       Bucket_Findings* found, u64* verdict)
{
    static std::atomic<bool> configured[64];
    if(!configured[ctx->device & 63])
    {
        CSA_CUDA(ctx, cudaFuncSetAttribute(bucket_counts_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(4u << BUCKET_MAX_BITS)));
        configured[ctx->device & 63] = true;
    }
    bucket_counts_kernel<<<unsigned(std::min<u64>(148, div_up(n, 2 * COUNT_BLOCK * COUNT_UNROLL))), COUNT_BLOCK, size_t(4) << bits, ctx->stream>>>(keys, n, begin_bit, end_bit, bits,
                                                                                                                                             least_digits, starts, found);
    CSA_LAUNCH_CHECK(ctx);
    launch_early(bucket_plan_kernel, 1, 1024, 0, ctx->stream, starts, u32(n), begin_bit, end_bit, bits, low_bits, least_digits, low_base, high_base, found, verdict);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}

int launch_bucket_sort(csa_ctx* ctx, const u64* kin, u64* kout, const void* vin, void* vout, u32 val_bytes, const u32* starts, u32 buckets, u64 n, u64 largest, Bucket_Findings* found,
                       int begin_bit, int top)
{
    if(val_bytes == 4) return launch_buckets_of<u32>(ctx, kin, kout, static_cast<const u32*>(vin), static_cast<u32*>(vout), starts, buckets, n, largest, found, begin_bit, top);
    return launch_buckets_of<u64>(ctx, kin, kout, static_cast<const u64*>(vin), static_cast<u64*>(vout), starts, buckets, n, largest, found, begin_bit, top);
}
