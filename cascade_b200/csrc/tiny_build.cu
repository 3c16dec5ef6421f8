// The suffix array of a text that one block holds in shared memory, in one launch. A build of a few thousand symbols by prefix_sort.cu's
// kernels is launches and read-backs (3001 tokens: 60 us of kernels in a call of 107 us); this way a call takes 36 us, 15 of them in the kernel (8000
// tokens: 108 and 44 us, 16000: 117 and 58 us).
//
// The symbols become their ranks among those that occur (a bit per symbol, and the bits before), so that nothing is as long as the alphabet. Every
// suffix gets a number f that never falls from a suffix to a greater one and is nearly even over the text's suffixes: the arithmetic code of its first
// symbols, from the exact counts, as far as 32 bits tell them apart. The suffixes are dealt into bins by f, a few bins for every suffix in short
// texts and one in the longest; inside a bin they are ordered by f, and where that is the same, by the text itself. A text with many suffixes in one
// bin, or with repeats that would take long to compare, is left to the general build: nothing has been written then.
#include "common.cuh"
#include "tiny_build.cuh"

#include <atomic>

namespace
{

constexpr int BLOCK = 1024, PER_MAX = int(TINY_BUILD_MAX / BLOCK);
constexpr u32 CODE_SYMBOLS = 24;    // symbols that f looks at, at most
constexpr u32 LONG_BIN = 64;        // suffixes of a bin at most
constexpr u32 MOST_PAIRS = 3u << 15;    // pairs of suffixes in one bin at most, of all bins: an even text has two a suffix. (16000 symbols of phrases that occur forty times, 33 a
                                        // suffix: compared all the same 642 us, left to the general build 221.)
constexpr u32 MOST_STEPS = 512, LEAST_STEPS = 32;       // of comparisons, four symbols each: what a warp may come to by what it has done, and from when on that is looked at
constexpr int MAX_BIN_BITS = 14;

constexpr u32 MAX = u32(TINY_BUILD_MAX);
constexpr u32 TEXT_AT = 0;
constexpr u32 CODE_AT = TEXT_AT + (MAX + 8) * 2;
constexpr u32 BIN_AT = CODE_AT + MAX * 4, BINS_MAX = 1u << MAX_BIN_BITS;
constexpr u32 F_AT = BIN_AT + (BINS_MAX + 8) * 2;
constexpr u32 DEALT_AT = F_AT + MAX * 4;
constexpr size_t TINY_SMEM = DEALT_AT + MAX * 2;
static_assert(TINY_SMEM + 1024 <= 227 * 1024 && CODE_AT % 16 == 0 && BIN_AT % 16 == 0 && F_AT % 16 == 0 && DEALT_AT % 16 == 0, "what a block has");
static_assert(MAX <= 16384 && CSA_MAX_PARTITIONS * 4 <= MAX * 2, "16-bit places; the partitions' sizes lie behind the order");
static_assert(65536 / 8 + 65536 / 32 * 2 <= MAX * 4, "the symbols' bits and their sums lie where f does later");

__device__ __forceinline__ u32 inclusive(u32 v)
{
    #pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const u32 t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if(int(lane_id()) >= o) v += t;
    }
    return v;
}

// Exclusive sum over the block. Ends without a barrier: the next call needs one before it.
__device__ __forceinline__ u32 exclusive(const u32 v, u32* warp_tot)
{
    const u32 inc = inclusive(v), warp = threadIdx.x >> 5;
    if(lane_id() == 31) warp_tot[warp] = inc;
    __syncthreads();
    return __reduce_add_sync(0xFFFFFFFFu, lane_id() < warp ? warp_tot[lane_id()] : 0u) + inc - v;
}

// A bit for each of four symbols, set where a and b differ. Behind the text there are symbols, too.
__device__ __forceinline__ u32 differences(const u16* a, const u16* b)
{
    u32 differ = 0;
    #pragma unroll
    for(u32 j = 0; j < 4; ++j) differ |= a[j] != b[j] ? 1u << j : 0u;
    return differ;
}

// One block; what bounds it is the chain of its steps and, near the longest text, their instructions.
// bucket_bits: the statistics tell partitions by as many leading bits of f. result: pinned host memory.
__global__ void __launch_bounds__(BLOCK) tiny_build_kernel(const u16* __restrict__ text, const u32 n, u8* __restrict__ sa40, const u32 p, const int bucket_bits, const u64* __restrict__ status,
                                                          Tiny_Result* __restrict__ result)
{
    extern __shared__ __align__(16) unsigned char smem[];
    u16* const T = reinterpret_cast<u16*>(smem + TEXT_AT);
    u32* const code = reinterpret_cast<u32*>(smem + CODE_AT);       // by rank of the symbol: counts, then 2^16 * (symbols before, its own) / n, 16 bits each
    u16* const start = reinterpret_cast<u16*>(smem + BIN_AT);       // counts of the bins, then their starts
    u32* const F = reinterpret_cast<u32*>(smem + F_AT);             // by bin: f, and
    u16* const dealt = reinterpret_cast<u16*>(smem + DEALT_AT);     // the suffix
    u32* const bits = F;                                            // a bit per symbol that occurs
    u16* const bits_before = reinterpret_cast<u16*>(bits + 2048);   // per word
    u16* const order = reinterpret_cast<u16*>(code);                // the array, once the code is no longer needed
    u32* const part = reinterpret_cast<u32*>(order + MAX);
    u16* const further_ones = order + MAX;                          // before that: places in the bins of suffixes that are not told apart yet
    __shared__ u32 warp_tot[BLOCK / 32];
    __shared__ u32 s_tied, s_partitions, s_most, s_symbols, s_pairs, s_further;
    __shared__ volatile u32 s_left;
    const u32 tid = threadIdx.x, lane = lane_id();
    const int bin_bits = min(MAX_BIN_BITS, 34 - __clz(n));          // two to eight bins for every suffix, one in the longest texts
    const u32 bins = 1u << bin_bits;

    const uint4 none = make_uint4(0, 0, 0, 0);
    if(tid < 512) reinterpret_cast<uint4*>(bits)[tid] = none;
    for(u32 i = tid; i < bins * 2 / 16 + 1; i += BLOCK) reinterpret_cast<uint4*>(start)[i] = none;
    for(u32 i = tid; i < (n + 3) / 4; i += BLOCK) reinterpret_cast<uint4*>(code)[i] = none;
    if(tid == 0) { s_tied = 0; s_partitions = 0; s_most = 0; s_pairs = 0; s_left = 0; s_further = 0; }
    for(u32 i = tid; i < (n + 7) / 8; i += BLOCK) reinterpret_cast<uint4*>(T)[i] = __ldg(reinterpret_cast<const uint4*>(text) + i);      // the text is padded
    __syncthreads();
    for(u32 i = tid; i < n; i += BLOCK)
    {
        const u32 a = T[i], bit = 1u << (a & 31);
        if((bits[a >> 5] & bit) == 0) atomicOr(bits + (a >> 5), bit);       // a frequent symbol's is there as a rule
    }
    __syncthreads();
    {
        const u32 a = __popc(bits[2 * tid]), b = __popc(bits[2 * tid + 1]), before = exclusive(a + b, warp_tot);
        reinterpret_cast<u32*>(bits_before)[tid] = before | (before + a) << 16;
        if(tid == BLOCK - 1) s_symbols = before + a + b;
    }
    __syncthreads();
    for(u32 i = tid; i < n; i += BLOCK)
    {
        const u32 a = T[i], r = bits_before[a >> 5] + __popc(bits[a >> 5] & ((1u << (a & 31)) - 1));
        T[i] = u16(r);
        atomicAdd(code + r, 1u);
    }
    __syncthreads();
    // A symbol that occurs gets four of 2^16 or more, so the ranges of different symbols never meet.
    {
        const u32 symbols = s_symbols, each = (symbols + BLOCK - 1) / BLOCK, first = tid * each, end = min(first + each, symbols);
        const u32 scale = n == 1 ? 0xFFFFFFFFu : u32((u64(1) << 32) / n);
        u32 sum = 0;
        for(u32 i = first; i < end; ++i) sum += code[i];
        u32 run = exclusive(sum, warp_tot), at = __umulhi(run << 16, scale);
        for(u32 i = first; i < end; ++i)
        {
            run += code[i];
            const u32 next = __umulhi(run << 16, scale);
            code[i] = at << 16 | ((next - at) & 0xFFFFu);           // 2^16, of a text of one symbol, leaves nothing: all suffixes meet in one bin
            at = next;
        }
    }
    __syncthreads();

    // f: the range of the first symbol, in it the range of the second, and so on until a range is too small to be told from its neighbours. Where that
    // is depends on the symbols read alone, so suffixes keep their order. A thread takes `per` suffixes side by side.
    u32 f[PER_MAX], rank[PER_MAX];      // rank: place in the bin, later in the bins' order
    #pragma unroll
    for(int i = 0; i < PER_MAX; ++i)
    {
        const u32 x = tid + i * BLOCK;
        if(x >= n) break;
        u32 low = 0, range = 0xFFFFFFFFu;
        for(u32 y = x, end = min(x + CODE_SYMBOLS, n); y < end && range >= 64; ++y)
        {
            const u32 c = code[T[y]];
            low += __umulhi(range, c & 0xFFFF0000u);
            range = __umulhi(range, c << 16);
        }
        f[i] = low;
        const u32 b = low >> (32 - bin_bits);
        const u32 old = atomicAdd(reinterpret_cast<u32*>(start) + (b >> 1), (b & 1) ? 0x10000u : 1u);
        rank[i] = (b & 1) ? old >> 16 : old & 0xFFFFu;
    }
    __syncthreads();

    // the bins' starts
    u32 longest = 0, tied = 0, pairs = 0;
    {
        constexpr int WORDS = int(BINS_MAX) / 2 / BLOCK;
        const u32 each = max(1u, bins / 2 / BLOCK), first = tid * each;
        u32* const words = reinterpret_cast<u32*>(start);
        u32 c[WORDS], sum = 0;
        #pragma unroll
        for(u32 k = 0; k < WORDS; ++k)
        {
            c[k] = k < each && first + k < bins / 2 ? words[first + k] : 0;
            const u32 a = c[k] & 0xFFFFu, b = c[k] >> 16;
            longest = __vmaxu2(longest, c[k]);
            tied += (a > 1 ? a : 0) + (b > 1 ? b : 0);
            pairs += a * a + b * b;         // below 2^32, as all bins' suffixes together are below 2^15
            sum += a + b;
        }
        u32 run = exclusive(sum, warp_tot);
        #pragma unroll
        for(u32 k = 0; k < WORDS; ++k)
            if(k < each && first + k < bins / 2)
            {
                words[first + k] = run * 0x10001u + (c[k] << 16);
                run += (c[k] & 0xFFFFu) + (c[k] >> 16);
            }
        if(tid == 0) start[bins] = u16(n);
        tied = __reduce_add_sync(0xFFFFFFFFu, tied);
        if(lane == 0 && tied) atomicAdd(&s_tied, tied);
        pairs = __reduce_add_sync(0xFFFFFFFFu, pairs);
        if(lane == 0) atomicAdd(&s_pairs, pairs);
    }
    bool left = __syncthreads_or(max(longest & 0xFFFFu, longest >> 16) > LONG_BIN) || s_pairs > MOST_PAIRS;
    if(!left)
    {
        #pragma unroll
        for(int i = 0; i < PER_MAX; ++i)
        {
            const u32 x = tid + i * BLOCK;
            if(x >= n) break;
            rank[i] += start[f[i] >> (32 - bin_bits)];
            dealt[rank[i]] = u16(x);
            F[rank[i]] = f[i];
        }
        __syncthreads();
        #pragma unroll
        for(int i = 0; i < PER_MAX; ++i)
        {
            const u32 x = tid + i * BLOCK;
            if(x >= n) break;
            const u32 b = f[i] >> (32 - bin_bits), s = start[b], e = start[b + 1];
            u32 place = s;
            bool further = false;           // eight symbols do not tell
            for(u32 k = s; k < e; ++k)
            {
                const u32 o = F[k];
                place += o < f[i];
                if(o != f[i] || k == rank[i]) continue;
                const u32 y = dealt[k], room = n - max(x, y);
                u32 differ = differences(T + x, T + y);
                if(differ == 0 && room > 4) differ = differences(T + x + 4, T + y + 4) << 4;
                const u32 l = differ ? __ffs(differ) - 1 : 8;
                if(l >= room) place += y > x;               // the shorter suffix comes first
                else if(differ) place += T[y + l] < T[x + l];
                else further = true;
            }
            if(further) further_ones[atomicAdd(&s_further, 1u)] = u16(rank[i]);
            else order[place] = u16(x);
        }
        __syncthreads();
        // The others, a thread to each wherever they stood: the lanes go through their bins and the comparisons side by side, so that they stay together.
        u32 steps = 0, done = 0;
        for(u32 first = tid - lane, count = s_further, rounds = (count - first + BLOCK - 1) / BLOCK; first < count; first += BLOCK, ++done)
        {
            const u32 q = first + lane;
            u32 r = 0, x = 0, mine = 0, s = 0, e = 0;
            if(q < count)
            {
                r = further_ones[q]; x = dealt[r]; mine = F[r];
                const u32 b = mine >> (32 - bin_bits);
                s = start[b]; e = start[b + 1];
            }
            u32 place = s;
            for(u32 t = 0, most = __reduce_max_sync(0xFFFFFFFFu, e - s); t < most; ++t)
            {
                const u32 k = s + t;
                u32 y = 0, room = 0, l = 0;
                bool same = false;
                if(k < e)
                {
                    const u32 o = F[k];
                    place += o < mine;
                    same = o == mine && k != r;
                    if(same) { y = dealt[k]; room = n - max(x, y); }
                }
                while(__any_sync(0xFFFFFFFFu, same && s_left == 0))         // s_left: the whole block leaves it, what is written from here on is not used
                {
                    if(++steps >= LEAST_STEPS && steps * rounds * most > MOST_STEPS * (done * most + t + 1)) s_left = 1;
                    if(!same) continue;
                    const u32 differ = differences(T + x + l, T + y + l);
                    l += differ ? __ffs(differ) - 1 : 4;
                    same = differ == 0 && l < room;
                    if(!same) place += l < room ? T[y + l] < T[x + l] : y > x;
                }
            }
            if(q < count) order[place] = u16(x);
        }
        __syncthreads();
        left = s_left != 0;
    }
    if(!left)
    {
        for(u32 i = tid; i < p; i += BLOCK) part[i] = 0;
        // 16 entries are 80 bytes
        const u32 first = tid * 16;
        if(first + 16 <= n)
        {
            const uint4 a = reinterpret_cast<const uint4*>(order)[2 * tid], b = reinterpret_cast<const uint4*>(order)[2 * tid + 1];
            const u32 v2[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            u32 w[20];
            #pragma unroll
            for(int j = 0; j < 20; ++j) w[j] = 0;
            #pragma unroll
            for(int e = 0; e < 16; ++e)
            {
                const u32 v = (e & 1) ? v2[e >> 1] >> 16 : v2[e >> 1] & 0xFFFFu;
                const int at = 5 * e, wi = at >> 2, sh = (at & 3) * 8;
                w[wi] |= v << sh;
                if(sh > 16) w[wi + 1] |= v >> (32 - sh);
            }
            uint4* const out = reinterpret_cast<uint4*>(sa40 + first * 5);
            #pragma unroll
            for(int j = 0; j < 5; ++j) out[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        }
        const u32 whole = n / 16 * 16;
        if(tid < (n - whole) * 5)
        {
            const u32 v = order[whole + tid / 5], byte = tid % 5;
            sa40[whole * 5 + tid] = byte < 2 ? u8(v >> (8 * byte)) : u8(0);
        }
        __syncthreads();
        // the statistics' partitions: a bucket belongs to the p-th part of the suffix array in which it starts
        if(tid < (1u << bucket_bits))
        {
            const u32 a = start[tid << (bin_bits - bucket_bits)], b = start[(tid + 1) << (bin_bits - bucket_bits)];
            if(b > a) atomicAdd(&part[u64(a) * p / n], b - a);
        }
        __syncthreads();
        u32 formed = 0, most = 0;
        for(u32 i = tid; i < p; i += BLOCK) { formed += part[i] != 0; most = max(most, part[i]); }
        if(formed) { atomicAdd(&s_partitions, formed); atomicMax(&s_most, most); }
    }
    __syncthreads();
    if(tid == 0)
    {
        result->tied = s_tied;
        result->partitions = s_partitions;
        result->max_partition = s_most;
        result->status = *status;
        result->done = left ? 0u : 1u;
    }
}

}   // namespace

int launch_tiny_build(csa_ctx* ctx, const u16* text, u64 n, u8* sa40, u32 p, int bucket_bits, Tiny_Result* result)
{
    if(n == 0 || n > TINY_BUILD_MAX) return csa_fail(ctx, CSA_E_LIMIT, "build: the text does not fit a block");
    static std::atomic<bool> configured[64];
    if(!configured[ctx->device & 63])
    {
        CSA_CUDA(ctx, cudaFuncSetAttribute(tiny_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(TINY_SMEM)));
        configured[ctx->device & 63] = true;
    }
    tiny_build_kernel<<<1, BLOCK, TINY_SMEM, ctx->stream>>>(text, u32(n), sa40, p, bucket_bits, ctx->d_status, result);
    CSA_LAUNCH_CHECK(ctx);
    return CSA_OK;
}
