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
template <int BLOCK, int BLOCKS, typename V>
__global__ void __launch_bounds__(BLOCK, BLOCKS) bucket_sort_kernel(const u64* __restrict__ keys_in, u64* __restrict__ keys_out, const V* __restrict__ vals_in,
                                                                   V* __restrict__ vals_out, const u32* __restrict__ starts, const u32 n, const u64 compared, const int top,
                                                                   const int begin)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr u32 CAP = BUCKET_CAP<BLOCK>;
    constexpr int ITEMS = BUCKET_ITEMS;
    u64* const stage = reinterpret_cast<u64*>(smem_raw);            // [CAP]
    u32* const bin = reinterpret_cast<u32*>(stage + CAP);           // [CAP / 2 + 8]: two 16-bit counters a word, then the bins' starts
    u16* const start = reinterpret_cast<u16*>(bin);
    u16* const from = reinterpret_cast<u16*>(bin + CAP / 2 + 8);    // [CAP]: the record's place in the bucket before
    V* const vals = reinterpret_cast<V*>(stage + CAP);              // [CAP], once the bins are no longer needed
    __shared__ u32 warp_tot[BLOCK / 32], s_differ[2];
    static_assert(BLOCK / 32 * 256 <= CAP && BLOCK >= 256 && ITEMS * 32 == 256 && CAP <= 8192, "the warps' counts lie where the bins do; places take 13 bits");
    const u32 tid = threadIdx.x;
    const u32 base = starts ? starts[blockIdx.x] : 0, m = (starts ? starts[blockIdx.x + 1] : n) - base;
    if(m == 0 || m > CAP) return;       // the host has seen to it that all fit
    keys_in += base; keys_out += base;
    if(vals_in != nullptr) { vals_in += base; vals_out += base; }

    const int bin_bits = min(32 - __clz(m - 1 | 1u), top - begin);  // bins: a power of two, at most CAP
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
        constexpr int WORDS = CAP / 2 / BLOCK;          // 4 words, 8 bins a thread
        u32 c[WORDS], sum = 0;
        const bool any = tid * WORDS * 2 <= bins;       // the words up to a multiple of WORDS were cleared
        if(any)
        {
            const uint4 v = reinterpret_cast<const uint4*>(bin)[tid];
            c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
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
                c[k] = a;
            }
            reinterpret_cast<uint4*>(bin)[tid] = make_uint4(c[0], c[1], c[2], c[3]);
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

template <typename V>
int launch_buckets_of(csa_ctx* ctx, const u64* kin, u64* kout, const V* vin, V* vout, const u32* starts, u32 buckets, u64 n, u64 largest, int begin, int top)
{
    const u64 compared = (top >= 64 ? ~0ull : (1ull << top) - 1) & (~0ull << begin);
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

int launch_bucket_sort(csa_ctx* ctx, const u64* kin, u64* kout, const void* vin, void* vout, u32 val_bytes, const u32* starts, u32 buckets, u64 n, u64 largest, int begin_bit,
                       int top)
{
    if(val_bytes == 4) return launch_buckets_of<u32>(ctx, kin, kout, static_cast<const u32*>(vin), static_cast<u32*>(vout), starts, buckets, n, largest, begin_bit, top);
    return launch_buckets_of<u64>(ctx, kin, kout, static_cast<const u64*>(vin), static_cast<u64*>(vout), starts, buckets, n, largest, begin_bit, top);
}
