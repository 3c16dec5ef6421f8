// The build of a whole suffix array on one GPU with text and all intermediates resident in HBM:
//   1. the suffixes sorted by the first bits of their encoded symbols (prefix_sort.cu);
//   2. the tied ones ordered group by group: first by their symbols, a few words of text at a time, then, where long repeats
//      leave ties, by the ranks of the suffixes h symbols further on, h doubling (refine.cu); groups of more than SMALL_GROUP
//      suffixes go through the radix sort and the rank kernels of doubling.cu;
//   3. 5-byte output.
//
// It stands for GPU_SACA::build_SA (src/GPU_SACA.cu:124-216): select_pivots (:290), partition (:737), initial_rank
// (:1052), exponentiate_prefix (:1998) and concatenate_partitions (:2167), for a text that fits the device.
#include "common.cuh"
#include "part.cuh"
#include "prefix_sort.cuh"
#include "refine.cuh"
#include "sort.cuh"
#include "tiny_build.cuh"

#include <algorithm>
#include <chrono>
#include <cstdlib>

namespace
{

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

struct Build_Layout
{
    size_t rec, sa, isa, tables, total;     // held by every build
    size_t sort_ws, scratch, work, more;    // held once ties have to be ranked (`more` bytes together)
};

Build_Layout layout_for(u64 n)
{
    Build_Layout L;
    L.rec = align256(n * 8);
    L.sa = align256(n * 4 + 64);
    L.isa = align256(n * 4);
    L.tables = align256(prefix_sort_table_bytes(prefix_sort_plan(n)));
    L.total = 2 * L.rec + L.sa + L.tables + 4096;
    L.sort_ws = align256(csa_sort_workspace_bytes(n));
    L.scratch = oversize_scratch_bytes(n);
    L.work = oversize_work_bytes(n);
    L.more = L.isa + L.sort_ws + L.scratch + L.work + 4096;
    return L;
}

// From here on a host build is done in four parts, so that the array's copy to the host (9.1 of the 15.6 ms of 1e8 suffixes) runs under
// the sorting: 13.7 to 14.4 ms (2e9: 0.27 to 0.33 s by box, 0.26 of them copies). Below it the parts' launches cost what the overlap gives.
constexpr u64 HOST_PARTS_MIN = u64(1) << 23;
// Up to here the local sort and the ties by text write 5-byte entries themselves. It spares a pass and a launch but costs instructions, which bound the local
// sort: 2^24 tokens 573 us without and 557 with it, 2e8 4.56 and 4.53 ms, 2e9 47.2 and 47.4 ms, and a text that is ranked has to be unpacked.
constexpr u64 PACKED_MAX = u64(1) << 25;
// Tied suffixes from which on (and a quarter of the text) groups are looked through for followers. Below, a generation costs its launches: near-duplicates of
// 10^6 tokens took 657 us without and 740 with it.
constexpr u64 FOLLOWED_MIN = u64(1) << 22;
// Large groups are ranked ahead of the small ones where they hold no more than one in LARGE_SHARE of their suffixes, as most of them share a few frequent symbols
// only: every step tells depth0 symbols or more, and is the last if it leaves more than three quarters.
// 1e9 near-duplicate suffixes with 1849 of them in large groups: 365 ms with the large groups left to the generations, so that nothing followed, 252 this way.
constexpr u64 LARGE_SHARE = 8;
constexpr u32 LARGE_STEPS = 12;
// And only where ranks pay, which a sample tells: nearly all suffixes have a follower, or most have and many share more symbols than the text is compared for, which need ranks
// anyway. Else most ties are settled by the text alone. ms a build of 4e8 suffixes, ranked and by text, in brackets the sample's two shares: phrases that occur four times, of 4 symbols
// (0.51, 0) 47.9 and 31.1, of 8 (0.83, 0) 42.7 and 39.7, of 12 (0.89, 0) 42.3 and 42.6, of 30 (0.96, 0) 42.1 and 46.1; near-duplicates with 1.3 % of their symbols replaced (0.76, 0.27)
// 84.7 and 100.6, with 2 % (0.67, 0.14) 115 and 99. Up to 2^24 suffixes, whose ranks stay in L2, three quarters are enough: 1.2e7 suffixes, phrases of 4 symbols 1.44 and
// 1.12 ms, of 7 (0.80, 0) 1.21 and 1.32.
bool ranks_pay(const Build_Counts& c, const u64 n)
{
    return u64(c.lead_on) * 8 >= u64(c.looked_at) * (n <= (u64(1) << 24) ? 6 : 7) || (u64(c.lead_on) * 10 >= u64(c.looked_at) * 7 && u64(c.far_ties) * 5 >= c.looked_at);
}

int set_build_count(csa_ctx* ctx, u32* at, u32 value)
{
    if(value == 0) CSA_CUDA(ctx, cudaMemsetAsync(at, 0, 4, ctx->stream));
    else CSA_CUDA(ctx, cudaMemcpyAsync(at, &value, 4, cudaMemcpyHostToDevice, ctx->stream));     // pageable: copied before the call returns
    return CSA_OK;
}

struct Build
{
    csa_ctx* ctx;
    const u16* T;
    u64 n;
    Build_Layout L;
    Prefix_Sort ps;
    Prefix_Tables tab;
    u64* front;         // the buffer with the current list: small groups from its front, large ones from its back
    u64* other;
    u32* sa;
    Build_Counts* counts;
    u64 small = 0, large = 0;
    // once ranks are needed
    u32* isa = nullptr;
    void* sort_ws = nullptr;
    u32* scratch = nullptr;
    u8* work = nullptr;
    // Large groups as the last generation left them, `large` entries in arrays instead of the buffer's back (see generation)
    bool in_arrays = false;
    u64 array_cap = 0;
    u32* head = nullptr;
    u32* pos = nullptr;
    u32* pos_other = nullptr;

    bool ranked = false;        // isa holds every suffix's rank

    u64* large_list(u64* buf) const { return buf + (n - large); }
    u32* ranks() const { return ranked ? isa : nullptr; }

    int read_counts(Build_Counts& c) { return read_build_counts(ctx, n, c); }

    int set_count(u32 Build_Counts::*field, u32 value) { return set_build_count(ctx, &(counts->*field), value); }

    // The buffers for ranking, from the context's second buffer.
    int more_memory()
    {
        if(isa) return CSA_OK;
        void* p = nullptr;
        CSA_TRY(csa_aux(ctx, L.more, &p));
        Carver cv(p, L.more);
        isa = cv.take<u32>(L.isa / 4);
        sort_ws = cv.take<u8>(L.sort_ws);
        scratch = cv.take<u32>(L.scratch / 4);
        work = cv.take<u8>(L.work);
        return cv.ok ? CSA_OK : csa_fail(ctx, CSA_E_NOMEM, "build: workspace too small");
    }

    // The few children of an ordinary text take buffers of their size; ranking, if it comes to that, asks for its own then.
    int sort_oversize(const Build_Counts& c)
    {
        const u64 few = n / OVERSIZE_SHARE;
        if(c.oversize_records > few)
        {
            CSA_TRY(more_memory());
            return sort_oversize_children(ctx, ps, tab, c, n, front, other, sa, counts, {sort_ws, L.sort_ws, scratch, work, L.work});
        }
        const size_t bytes = oversize_buffers_bytes(few);
        void* p = nullptr;
        CSA_TRY(csa_aux(ctx, bytes, &p));
        return sort_oversize_children(ctx, ps, tab, c, n, front, other, sa, counts, oversize_buffers(p, few));
    }

    int check_large_depth(const Build_Counts& c, u64 depth0)
    {
        if(c.large_depth < depth0 || c.large_depth > u64(ps.key_bits)) return csa_fail(ctx, CSA_E_DEVICE, "build: the large groups' depth is out of range");
        return CSA_OK;
    }

    // One generation of prefix doubling: the suffixes of every group ordered by the ranks of those h symbols further on. The first
    // `idle` entries of the list share more than h symbols already and stay as they are.
    //
    // What is left of the large groups is counted by size. Where few of them have become small (up to one in eight), they all stay in the arrays
    // that the ranking left, and the radix sort takes the small ones once more: to write the two lists and read them again costs 40 bytes a
    // suffix, a suffix too many in a radix sort some 200.
    int generation(u64 h, u64 idle)
    {
        const bool all_by_sort = h > MAX_SMALL_H;       // small groups compare 32-bit numbers, which need h below that
        const u64 ns = all_by_sort ? 0 : small - idle, nl = large + (all_by_sort ? small - idle : 0);
        if(!in_arrays) array_cap = nl;
        const size_t one = align256(array_cap * 4);
        if(nl > array_cap || align256(ns * 4) + 3 * one > L.work) return csa_fail(ctx, CSA_E_NOMEM, "build: workspace too small");
        u32* const secs = reinterpret_cast<u32*>(work);         // the arrays lie at the end: they stay where they are while this one grows and shrinks
        if(!in_arrays)
        {
            u8* const arrays = work + L.work - 3 * one;
            head = reinterpret_cast<u32*>(arrays); pos = reinterpret_cast<u32*>(arrays + one); pos_other = reinterpret_cast<u32*>(arrays + 2 * one);
        }
        Isa_View iv{};
        iv.shard[0] = isa; iv.shard_size = n; iv.gpus = 1;
        // every rank that this generation reads is read before any is written
        CSA_TRY(launch_gather_ranks(ctx, front + idle, ns, isa, n, h, secs));
        // behind what refine_by_ranks writes, on a 16-byte boundary where there is room: the sort and the ranking then load two keys at once
        const u64 keys_at = (n - nl) - ((n - nl) & (n - nl > idle + ns ? 1 : 0));
        u64* const keysA = other + keys_at;
        u64* const keysB = front + keys_at;
        const int sec_bits = bits_for(n - 1 + h), prim_bits = std::max(1, bits_for(n - 1));
        if(nl)
        {
            if(sec_bits + prim_bits > 64) return csa_fail(ctx, CSA_E_LIMIT, "build: rank pair does not fit a 64-bit key");
            if(all_by_sort) CSA_TRY(launch_unpack_list(ctx, front + idle, small - idle, head + large, pos + large));
            if(!in_arrays) CSA_TRY(launch_unpack_list(ctx, large_list(front), large, head, pos));
            CSA_TRY(launch_keys_gen(ctx, head, pos, nl, n, h, sec_bits, iv, keysA));
        }
        if(idle) CSA_CUDA(ctx, cudaMemcpyAsync(other, front, idle * 8, cudaMemcpyDeviceToDevice, ctx->stream));
        CSA_TRY(set_count(&Build_Counts::next_small, u32(idle)));
        CSA_TRY(set_count(&Build_Counts::large, 0));
        CSA_TRY(launch_refine_by_ranks(ctx, front + idle, ns, secs, isa, sa, other, counts));
        Build_Counts c;
        if(nl)
        {
            int in_alt = 0;
            CSA_TRY(csa_sort_pairs(ctx, reinterpret_cast<uint64_t*>(keysA), reinterpret_cast<uint64_t*>(keysB), pos, pos_other, 4, nl, 0, sec_bits + prim_bits, sort_ws, L.sort_ws, &in_alt));
            u64* const ks = in_alt ? keysB : keysA;
            u64* const upd = in_alt ? keysA : keysB;
            if(in_alt) std::swap(pos, pos_other);       // pos: the sorted positions; the tied ones go to the other array
            CSA_CUDA(ctx, cudaMemsetAsync(ctx->d_scalars, 0, 8, ctx->stream));
            const Slot_Map whole{nullptr, nullptr, 0, 0};
            CSA_TRY(launch_rank_and_compact(ctx, ks, pos, nl, sec_bits, 0, iv, whole, sa, head, pos_other, ctx->d_scalars, scratch, upd, false));
            std::swap(pos, pos_other);
            CSA_TRY(apply_updates_in_address_order(ctx, isa, upd, ks, nl, bits_for(n - 1), sort_ws, L.sort_ws));
            CSA_TRY(launch_count_by_size(ctx, head, nl, ctx->d_scalars, counts, scratch));
        }
        CSA_TRY(read_counts(c));
        small = c.next_small; large = c.large;
        in_arrays = nl != 0 && large != 0 && 2 * h <= MAX_SMALL_H && u64(c.now_small) * 8 <= u64(c.now_small) + c.large;
        if(in_arrays) { small -= c.now_small; large += c.now_small; }
        else if(nl) CSA_TRY(launch_split_by_size(ctx, head, pos, nl, ctx->d_scalars, other, n, scratch));
        std::swap(front, other);
        return CSA_OK;
    }

    // The same of the ends of rows of groups that follow one another (refine.cu).
    int generation_of_ends(u64 h, const u32* bits)
    {
        CSA_TRY(set_count(&Build_Counts::next_small, 0));
        CSA_TRY(launch_refine_ends(ctx, front, small, h, reinterpret_cast<u64*>(work), bits, isa, n, sa, other, counts));
        Build_Counts c;
        CSA_TRY(read_counts(c));
        small = c.next_small;
        std::swap(front, other);
        return CSA_OK;
    }
};

// The whole build in one block, where the text fits one and is not repetitive (done). The counters come straight into pinned memory.
int build_in_one_block(csa_ctx* ctx, const u16* T, const u64 n, u32 p, u8* sa40, csa_build_stats& st, bool& done)
{
    Tiny_Result* const result = reinterpret_cast<Tiny_Result*>(ctx->h_scalars + CSA_COUNTS_WORD);
    cudaEvent_t* const ev = ctx->phase_event;
    CSA_TRY(launch_tiny_build(ctx, T, n, sa40, p, prefix_sort_plan(n).b2, result));
    CSA_CUDA(ctx, cudaEventRecord(ev[4], ctx->stream));
    CSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if(result->status != 0) { u64 b = 0; return csa_sync(ctx, reinterpret_cast<uint64_t*>(&b)); }
    done = result->done != 0;
    if(!done) return CSA_OK;
    st.partitions = result->partitions;
    st.max_partition = result->max_partition;
    st.active_after_gen0 = result->tied;
    if(result->tied) { st.generations = 1; st.active_per_gen[0] = result->tied; }
    ctx->counters[1] += 1;
    ctx->counters[2] += n;
    float ms = 0;
    cudaEventElapsedTime(&ms, ev[0], ev[4]);
    st.ms_gen0 = st.ms_total = ms;
    return CSA_OK;
}

int build_core(csa_ctx* ctx, const u16* T, const u64 n, u32 p, const u64 seed, u8* sa40, csa_build_stats* stats, void* ws, size_t ws_bytes)
{
    (void)seed;         // drives the sampling of splitters in the sharded and part-at-a-time builds; this build's sample is the same for all seeds
    csa_build_stats local_stats;
    csa_build_stats& st = stats ? *stats : local_stats;
    std::memset(&st, 0, sizeof(st));
    st.n = n;
    const u64 launches_before = ctx->counters[0], passes_before = ctx->counters[1], records_before = ctx->counters[2];
    const bool debug = std::getenv("CSA_DEBUG") != nullptr;

    for(auto& e : ctx->phase_event) if(!e) CSA_CUDA(ctx, cudaEventCreate(&e));
    cudaEvent_t* const ev = ctx->phase_event;
    CSA_CUDA(ctx, cudaEventRecord(ev[0], ctx->stream));

    if(n <= TINY_BUILD_MAX)
    {
        bool done = false;
        CSA_TRY(build_in_one_block(ctx, T, n, p, sa40, st, done));
        if(done)
        {
            st.kernel_launches = ctx->counters[0] - launches_before;
            st.sort_passes = ctx->counters[1] - passes_before;
            st.sort_records = ctx->counters[2] - records_before;
            return CSA_OK;
        }
    }

    Build b{ctx, T, n, layout_for(n), prefix_sort_plan(n)};
    Carver cv(ws, ws_bytes);
    u64* recA = cv.take<u64>(b.L.rec / 8);
    u64* recB = cv.take<u64>(b.L.rec / 8);
    b.sa = cv.take<u32>(b.L.sa / 4);
    if(!cv.ok || !prefix_sort_carve(cv, b.ps, b.tab)) return csa_fail(ctx, CSA_E_NOMEM, "build: workspace too small");
    b.counts = reinterpret_cast<Build_Counts*>(ctx->d_scalars + CSA_COUNTS_WORD);
    const Ties_In_Any_Order free_ties(ctx);     // ties of the radix sorts are resolved by what follows them

    // ---- generation 0, and the ties that it leaves by their symbols --------------------------------------------------------
    // A short build writes its output as positions are found; ranking, if it comes to that, makes 4-byte positions from it.
    u32* words = n > PACKED_MAX ? b.sa : nullptr;       // b.sa, once the positions are there; the output else
    CSA_TRY(launch_prefix_sort(ctx, b.ps, b.tab, T, recA, recB, words, sa40, p, b.counts, &b.front, &b.other, ev[1]));
    CSA_CUDA(ctx, cudaEventRecord(ev[2], ctx->stream));
    const u64 depth0 = shared_symbols(b.ps);
    u64 depth = TEXT_DEPTH;
    // More tied suffixes than this are first looked through for groups that follow one another: those need not be compared.
    const u64 most_by_text = std::max(FOLLOWED_MIN, n / 4);
    Build_Counts c;
    CSA_TRY(launch_refine_by_text(ctx, T, n, depth0, depth, b.front, b.other, words, sa40, nullptr, b.counts, n, most_by_text, b.tab.code, b.ps.key_bits));
    bool done = false;          // the output is complete, and the events have been waited for with the counters below
    if(!words)
    {
        CSA_CUDA(ctx, cudaEventRecord(ev[3], ctx->stream));
        CSA_CUDA(ctx, cudaEventRecord(ev[4], ctx->stream));
        done = true;
    }
    CSA_TRY(b.read_counts(c));
    if(c.oversize)
    {
        done = false;
        if(debug) std::fprintf(stderr, "[csa] %u children (%u suffixes) do not fit a block\n", c.oversize, c.oversize_records);
        CSA_TRY(b.sort_oversize(c));
        if(!words) CSA_TRY(launch_pack_oversize(ctx, b.tab, c.oversize, b.sa, sa40));
        CSA_TRY(launch_refine_by_text(ctx, T, n, depth0, depth, b.front, b.other, words, sa40, nullptr, b.counts, n, most_by_text, b.tab.code, b.ps.key_bits));
        CSA_TRY(b.read_counts(c));
    }
    st.partitions = c.partitions;
    st.max_partition = c.max_partition;
    st.active_after_gen0 = u64(c.small) + c.large;
    if(debug) std::fprintf(stderr, "[csa] n=%llu key bits %d: tied after generation 0: %u in small groups, %u in large ones; %u of %u batches crowded, %u runs left, %u of %u first batches uneven\n", n, b.ps.key_bits, c.small, c.large, c.crowded, c.batches, c.medium, c.tries & 0xFFFFu,
                           c.tries >> 16);
    u32 gen = 0;
    if(st.active_after_gen0) st.active_per_gen[gen++] = st.active_after_gen0;
    // The few large groups beside many small ones are ranked first, if some steps do it (LARGE_STEPS); a group that follows another is small.
    // Groups that lead, one symbol on, to a whole group again (refine.cu): where they hold half of the tied suffixes, the others alone go on, and they
    // take over their order at the end (near-duplicate documents: nineteen in twenty).
    u64 followed = 0;
    u64* ends_list = nullptr;           // all ends, as they were found
    u64 ends_found = 0;
    u32* bits = nullptr;
    u64 large_shared = 0;               // symbols that the large groups' suffixes share, once that has been found out
    if(c.small > most_by_text)
    {
        done = false;
        b.small = c.small;
        b.large = c.large;
        bool rank = c.large <= c.small / LARGE_SHARE && ranks_pay(c, n);
        if(debug) std::fprintf(stderr, "[csa] of %u tied suffixes looked at %u are tied one symbol on, %u share %llu symbols: %s\n", c.looked_at, c.lead_on, c.far_ties, depth,
                               rank ? "ranked" : "compared in the text");
        if(rank)
        {
            // Without the buffers the ties are compared in the text first: the ranks may not be needed then.
            const std::string err = ctx->err;
            const int rc = b.more_memory();
            if(rc != CSA_OK && rc != CSA_E_NOMEM) return rc;
            if(rc != CSA_OK) { ctx->err = err; rank = false; }
        }
        if(rank)
        {
            if(!words) CSA_TRY(launch_unpack_sa40(ctx, sa40, n, b.sa));
            words = b.sa;
            CSA_TRY(launch_make_inverse(ctx, b.sa, n, b.front, b.small, b.large_list(b.front), b.large, b.isa, reinterpret_cast<u64*>(b.work)));
            b.ranked = true;
            if(b.large)
            {
                CSA_TRY(launch_large_depth(ctx, b.large_list(b.front), b.large, T, n, b.tab.code, b.ps.key_bits, b.counts));
                CSA_TRY(b.read_counts(c));
                CSA_TRY(b.check_large_depth(c, depth0));
                large_shared = c.large_depth;
            }
            // Whatever the ranks tell apart: the small groups' suffixes share depth0 symbols at least.
            for(u32 step = 0; step < LARGE_STEPS && b.large; ++step)
            {
                const u64 before = b.large;
                if(gen < 48) st.active_per_gen[gen] = b.small + b.large;
                ++gen;
                CSA_TRY(b.generation(large_shared, b.small));
                if(debug) std::fprintf(stderr, "[csa] large groups, h=%llu: %llu -> %llu\n", large_shared, before, b.large);
                large_shared += depth0;
                if(b.large > before - before / 4) break;
            }
        }
        u64 ends = b.small;
        if(b.ranked && !b.large)
        {
            CSA_TRY(b.set_count(&Build_Counts::next_small, 0));
            bits = reinterpret_cast<u32*>(b.work + (b.L.work - follower_bits_bytes(n)) / 256 * 256);
            CSA_TRY(launch_split_followed(ctx, b.front, b.small, b.isa, n, reinterpret_cast<u32*>(b.work), b.sa, bits, b.other, b.counts));
            Build_Counts f;
            CSA_TRY(b.read_counts(f));
            if(u64(f.next_small) + f.large != b.small) return csa_fail(ctx, CSA_E_DEVICE, "build: the groups with and without a follower do not add up");
            if(debug) std::fprintf(stderr, "[csa] %u of %llu have a follower\n", f.large, b.small);
            if(2 * u64(f.large) >= b.small)
            {
                followed = f.large;
                ends = ends_found = f.next_small;
                ends_list = b.other + (n - ends);           // the lists that follow are no longer than half of the buffer
                CSA_CUDA(ctx, cudaMemcpyAsync(ends_list, b.other, ends * 8, cudaMemcpyDeviceToDevice, ctx->stream));
                std::swap(b.front, b.other);
            }
        }
        CSA_TRY(b.set_count(&Build_Counts::small, u32(ends)));
        CSA_TRY(b.set_count(&Build_Counts::next_small, 0));
        CSA_TRY(b.set_count(&Build_Counts::large, u32(b.large)));
        CSA_TRY(launch_refine_by_text(ctx, T, n, depth0, depth, b.front, b.other, words, sa40, b.ranks(), b.counts, ends, n));
        CSA_TRY(b.read_counts(c));
        c.large = u32(b.large);
    }
    b.large = c.large;
    if(b.large && !b.in_arrays) CSA_CUDA(ctx, cudaMemcpyAsync(b.large_list(b.other), b.large_list(b.front), b.large * 8, cudaMemcpyDeviceToDevice, ctx->stream));
    std::swap(b.front, b.other);
    b.small = c.next_small;
    // Few suffixes left, in small groups: reading on in the text costs less than an inverse array of the whole text.
    while(b.small && !b.large && !followed && b.small * depth <= n && depth < n)
    {
        done = false;
        if(gen < 48) st.active_per_gen[gen] = b.small;
        ++gen;
        CSA_CUDA(ctx, cudaMemcpyAsync(&b.counts->small, &b.counts->next_small, 4, cudaMemcpyDeviceToDevice, ctx->stream));
        CSA_TRY(b.set_count(&Build_Counts::next_small, 0));
        CSA_TRY(launch_refine_by_text(ctx, T, n, depth, 4 * depth, b.front, b.other, words, sa40, b.ranks(), b.counts, b.small, n));
        CSA_TRY(b.read_counts(c));
        if(debug) std::fprintf(stderr, "[csa] text up to symbol %llu: %llu -> %u\n", 4 * depth, b.small, c.next_small);
        std::swap(b.front, b.other);
        b.small = c.next_small;
        depth *= 4;
    }

    // ---- doubling generations -------------------------------------------------------------------------------
    if(b.small || b.large || followed)
    {
        done = false;
        CSA_TRY(b.more_memory());
        if(!words) CSA_TRY(launch_unpack_sa40(ctx, sa40, n, b.sa));
        words = b.sa;
        if(!b.ranked) CSA_TRY(launch_make_inverse(ctx, b.sa, n, b.front, b.small, b.large_list(b.front), b.large, b.isa, reinterpret_cast<u64*>(b.work)));
        u64 idle = b.large ? b.small : 0;               // in small groups already, hence ordered up to `depth`
        u64 shared = depth;                             // symbols that all others' groups share at least
        if(b.large)
        {
            // A large group was not compared in the text: it shares the whole symbols of generation 0's key. Frequent symbols, of which large groups
            // are made, have short code words, so that is more than what any key holds (depth0 = 1): one symbol repeated 2^24 times starts at 25
            // and takes 22 generations instead of 26.
            if(!large_shared)
            {
                CSA_TRY(launch_large_depth(ctx, b.large_list(b.front), b.large, T, n, b.tab.code, b.ps.key_bits, b.counts));
                CSA_TRY(b.read_counts(c));
                CSA_TRY(b.check_large_depth(c, depth0));
                large_shared = c.large_depth;
            }
            shared = std::min(large_shared, depth);
        }
        // Ranks tell `shared` symbols from any step of up to as many: doubling takes the longest step. Above 2^31 suffixes a step may be too long for
        // a sort key of two ranks (n - 1 + h has to fit beside bits_for(n - 1) bits in 64); steps of the longest that fits go on from there.
        const u64 longest_step = (u64(1) << (64 - bits_for(n - 1))) - n;
        while(b.small || b.large)
        {
            const u64 active = b.small + b.large + followed;
            if(idle && (shared >= depth || (idle == b.small && !b.large))) { shared = depth; idle = 0; }       // they join when the others have come as far
            if(gen < 48) st.active_per_gen[gen] = active;
            ++gen;
            const u64 h = followed ? shared : std::min(shared, longest_step);
            if(followed) CSA_TRY(b.generation_of_ends(h, bits));
            else CSA_TRY(b.generation(h, idle));
            if(debug) std::fprintf(stderr, "[csa] generation %u: h=%llu active %llu -> %llu (%llu in large groups)\n", gen, h, active, b.small + b.large, b.large);
            shared += h;
            if(shared > 2 * n + 2 * depth) return csa_fail(ctx, CSA_E_DEVICE, "build: doubling did not terminate");
        }
        if(followed) CSA_TRY(launch_place_followed(ctx, ends_list, ends_found, bits, b.isa, n, b.sa, reinterpret_cast<u64*>(b.work)));
    }
    st.generations = gen;

    // ---- output ------------------------------------------------------------------------------------------------
    if(!done)
    {
        CSA_CUDA(ctx, cudaEventRecord(ev[3], ctx->stream));
        if(words) CSA_TRY(launch_pack_sa40(ctx, b.sa, n, sa40));
        CSA_CUDA(ctx, cudaEventRecord(ev[4], ctx->stream));
        u64 bits = 0;
        CSA_TRY(csa_sync(ctx, reinterpret_cast<uint64_t*>(&bits)));
    }

    float ms = 0;
    cudaEventElapsedTime(&ms, ev[0], ev[1]); st.ms_partition = ms;
    cudaEventElapsedTime(&ms, ev[1], ev[2]); st.ms_gen0 = ms;
    cudaEventElapsedTime(&ms, ev[2], ev[3]); st.ms_doubling = ms;
    cudaEventElapsedTime(&ms, ev[3], ev[4]); st.ms_output = ms;
    cudaEventElapsedTime(&ms, ev[0], ev[4]); st.ms_total = ms;
    st.kernel_launches = ctx->counters[0] - launches_before;
    st.sort_passes = ctx->counters[1] - passes_before;
    st.sort_records = ctx->counters[2] - records_before;
    return CSA_OK;
}

int check_build_args(csa_ctx* ctx, const void* text, u64 n, u32 p, const void* out)
{
    if(!ctx || !text || !out) return csa_fail(ctx, CSA_E_INVALID, "build: null argument");
    if(n == 0) return csa_fail(ctx, CSA_E_INVALID, "build: empty text");
    if(p == 0 || p > CSA_MAX_PARTITIONS) return csa_fail(ctx, CSA_E_LIMIT, "build: partition count out of range");
    if(n >= (u64(1) << 32) - (u64(1) << 26)) return csa_fail(ctx, CSA_E_LIMIT, "build: this build addresses fewer than 2^32 - 2^26 suffixes per call");
    return CSA_OK;
}

}   // namespace

size_t oversize_scratch_bytes(u64 records) { return align256(div_up(records, RANK_TILE) * 3 * 4 + 256); }
size_t oversize_work_bytes(u64 records) { return align256(records * 12) + 16 * 256; }
size_t oversize_buffers_bytes(u64 records) { return align256(csa_sort_workspace_bytes(records)) + oversize_scratch_bytes(records) + oversize_work_bytes(records); }
Oversize_Buffers oversize_buffers(void* at, u64 records)
{
    const size_t sort_bytes = align256(csa_sort_workspace_bytes(records)), scratch_bytes = oversize_scratch_bytes(records);
    u8* const p = static_cast<u8*>(at);
    return {p, sort_bytes, reinterpret_cast<u32*>(p + sort_bytes), p + sort_bytes + scratch_bytes, oversize_work_bytes(records)};
}

int sort_oversize_children(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& tab, const Build_Counts& c, u64 n, u64* front, u64* other, u32* sa, Build_Counts* counts,
                           const Oversize_Buffers& b)
{
    const u64 M = c.oversize_records;
    if(M > n || u64(c.small) + c.large + M > n) return csa_fail(ctx, CSA_E_DEVICE, "build: oversize children do not add up");
    const Ties_In_Any_Order free_ties(ctx);
    u64* const keysA = front + c.small;
    u64* const keysB = other;
    Carver cv(b.work, b.work_bytes);
    u32* posA = cv.take<u32>(M);
    u32* posB = cv.take<u32>(M);
    u32* head = cv.take<u32>(M);
    if(!cv.ok) return csa_fail(ctx, CSA_E_NOMEM, "build: workspace too small");
    CSA_TRY(launch_gather_oversize(ctx, ps, tab, c.oversize, other, keysA, posA, b.scratch));
    int in_alt = 0;
    CSA_TRY(csa_sort_pairs(ctx, reinterpret_cast<uint64_t*>(keysA), reinterpret_cast<uint64_t*>(keysB), posA, posB, 4, M, 0, 64, b.sort_ws, b.sort_bytes, &in_alt));
    u64* const ks = in_alt ? keysB : keysA;
    CSA_CUDA(ctx, cudaMemsetAsync(ctx->d_scalars, 0, 8, ctx->stream));
    Isa_View none{};
    const Slot_Map whole{nullptr, nullptr, 0, 0};
    CSA_TRY(launch_rank_and_compact(ctx, ks, in_alt ? posB : posA, M, 32, 0, none, whole, sa, head, in_alt ? posA : posB, ctx->d_scalars, b.scratch, in_alt ? keysA : keysB, true));
    CSA_TRY(set_build_count(ctx, &counts->next_small, c.small));
    CSA_TRY(launch_count_by_size(ctx, head, M, ctx->d_scalars, counts, b.scratch));
    CSA_TRY(launch_split_by_size(ctx, head, in_alt ? posA : posB, M, ctx->d_scalars, front, n, b.scratch));
    CSA_CUDA(ctx, cudaMemcpyAsync(&counts->small, &counts->next_small, 4, cudaMemcpyDeviceToDevice, ctx->stream));
    CSA_TRY(set_build_count(ctx, &counts->next_small, 0));
    CSA_TRY(set_build_count(ctx, &counts->wide, 1));
    return set_build_count(ctx, &counts->oversize, 0);
}

extern "C" size_t csa_build_device_bytes(uint64_t n, uint32_t p)
{
    (void)p;
    const Build_Layout L = layout_for(n);
    return L.total + L.more + CSA_ALLOC_SLACK;
}

extern "C" int csa_build_sa(csa_ctx* ctx, const uint16_t* text, uint64_t n, uint32_t p, uint64_t seed, uint8_t* sa40, csa_build_stats* stats)
{
    CSA_TRY(check_build_args(ctx, text, n, p, sa40));
    if((reinterpret_cast<uintptr_t>(text) & 15) || (reinterpret_cast<uintptr_t>(sa40) & 15))
        return csa_fail(ctx, CSA_E_INVALID, "build: text and output must be 16-byte aligned");
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    const Build_Layout L = layout_for(n);
    const size_t bytes = L.total;
    void* ws = nullptr;
    CSA_TRY(csa_arena(ctx, bytes, &ws, L.more));
    return build_core(ctx, text, n, p, seed, sa40, stats, ws, bytes);
}

extern "C" int csa_build_sa_host(csa_ctx* ctx, const uint16_t* text_host, uint64_t n, uint32_t p, uint64_t seed, uint8_t* sa40_host, csa_build_stats* stats)
{
    CSA_TRY(check_build_args(ctx, text_host, n, p, sa40_host));
    CSA_CUDA(ctx, cudaSetDevice(ctx->device));
    const Build_Layout L = layout_for(n);
    const size_t core = L.total;
    const size_t text_bytes = align256((n + CSA_TEXT_PAD) * 2), out_bytes = align256(5 * n + CSA_SA_PAD_BYTES);
    const u16* text_at = text_host;
    if(n >= HOST_PARTS_MIN)
    {
        csa_build_stats local_stats;
        csa_build_stats& st = stats ? *stats : local_stats;
        std::memset(&st, 0, sizeof(st));
        st.n = n;
        const auto t_start = std::chrono::steady_clock::now();
        const u64 launches_before = ctx->counters[0], passes_before = ctx->counters[1], records_before = ctx->counters[2];
        void* p_text = nullptr;
        CSA_TRY(csa_aux(ctx, text_bytes, &p_text));         // the parts' buffers take the arena
        u16* const T = static_cast<u16*>(p_text);
        CSA_CUDA(ctx, cudaMemcpyAsync(T, text_host, n * 2, cudaMemcpyHostToDevice, ctx->stream));
        CSA_CUDA(ctx, cudaMemsetAsync(T + n, 0, CSA_TEXT_PAD * 2, ctx->stream));
        bool done = false;
        CSA_TRY(build_direct_parts(ctx, T, n, p, n / 4 + n / 64, sa40_host, st, done));
        if(done)
        {
            st.ms_total = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
            st.kernel_launches = ctx->counters[0] - launches_before;
            st.sort_passes = ctx->counters[1] - passes_before;
            st.sort_records = ctx->counters[2] - records_before;
            return CSA_OK;
        }
        text_at = T;        // repeats that need ranks: the whole build, from the copy on the device
    }
    const size_t bytes = core + text_bytes + out_bytes;
    void* ws = nullptr;
    CSA_TRY(csa_arena(ctx, bytes, &ws, L.more));
    u8* base = static_cast<u8*>(ws);
    u16* text_dev = reinterpret_cast<u16*>(base);
    u8* out_dev = base + text_bytes;
    CSA_CUDA(ctx, cudaMemcpyAsync(text_dev, text_at, n * 2, cudaMemcpyDefault, ctx->stream));
    CSA_CUDA(ctx, cudaMemsetAsync(text_dev + n, 0, CSA_TEXT_PAD * 2, ctx->stream));
    CSA_TRY(build_core(ctx, text_dev, n, p, seed, out_dev, stats, base + text_bytes + out_bytes, core));
    CSA_CUDA(ctx, cudaMemcpyAsync(sa40_host, out_dev, 5 * n, cudaMemcpyDeviceToHost, ctx->stream));
    CSA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return CSA_OK;
}
