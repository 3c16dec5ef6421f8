// Internal declarations of the steps that order tied suffixes after the initial sort of the resident build.
// A list holds (first slot of the group << 32) | position, group by group; small groups (up to SMALL_GROUP suffixes) fill a
// list's buffer from the front, large ones from the back.
#pragma once
#include "common.cuh"
#include "prefix_sort.cuh"

// Text is compared up to this depth before ranks are: past it one more doubling costs a suffix less (an inverse rank, 64 bytes of
// DRAM traffic) than its next symbols do.
constexpr u64 TEXT_DEPTH = 49;         // what tied suffixes share at least (1) + a wide round (refine.cu)

// The counters of the build as the stream leaves them; waits for the stream. Fails if a kernel reported an error or if the lists
// hold more than `most` entries.
int read_build_counts(csa_ctx* ctx, u64 most, Build_Counts& c);

// Orders the small groups of `list` by their suffixes' symbols [from, to) read straight from the text (a suffix that ends
// inside them comes before those that go on): every group that is left shares `to` symbols. Suffixes that are alone now go to
// their slots of sa or, where sa is null, as 5-byte entries to sa40, the others to next (front; counts->next_small entries). `expected`: about how many entries the list holds
// (its length is counts->small).
// A list of more than `most` entries is left alone; with the code given, about TIE_SAMPLE of its entries, spread over it, are looked at (counts->looked_at): those whose group
// is still tied one symbol on (lead_on; about the share that launch_split_followed finds to have a follower), and those that another of their group ties with up to symbol
// `to` (far_ties). isa (or null): every suffix's new rank goes there, too.
constexpr u32 TIE_SAMPLE = 1024;
int launch_refine_by_text(csa_ctx* ctx, const u16* T, u64 n, u64 from, u64 to, const u64* list, u64* next, u32* sa, u8* sa40, u32* isa, Build_Counts* counts, u64 expected, u64 most,
                          const u32* code = nullptr, int key_bits = 0);

// secs[i] = what the i-th entry of the list is ordered by in the generation that compares h symbols further on: the rank of the
// suffix h symbols on, or, where the text ends before, a smaller number that falls with the position.
constexpr u64 MAX_SMALL_H = u64(1) << 26;
int launch_gather_ranks(csa_ctx* ctx, const u64* list, u64 count, const u32* isa, u64 n, u64 h, u32* secs);
// Orders the small groups of the list by secs; new ranks go into isa, single suffixes into sa, the others to `next` behind the
// counts->next_small entries that are there.
int launch_refine_by_ranks(csa_ctx* ctx, const u64* list, u64 count, const u32* secs, u32* isa, u32* sa, u64* next, Build_Counts* counts);

// Groups whose suffixes lead, one symbol on, to a whole group again (refine.cu). The list's other groups, the ends, go to next
// (counts->next_small); counts->large receives the number of suffixes in groups that have a follower. Both counters start from 0. A group shares a symbol at least.
// bits: follower_bits_bytes(n), a bit per position, set for those suffixes; secs: a word per entry; the first slot of every group in sa receives its size. All groups are small and were ranked by isa.
inline size_t follower_bits_bytes(u64 n) { return align_up256((n / 64 + 2) * 8); }
int launch_split_followed(csa_ctx* ctx, const u64* list, u64 count, const u32* isa, u64 n, u32* secs, u32* sa, u32* bits, u64* next, Build_Counts* counts);
// One generation of the ends, h symbols on (they share as many): as launch_gather_ranks and launch_refine_by_ranks. secs: a double word per entry.
int launch_refine_ends(csa_ctx* ctx, const u64* list, u64 count, u64 h, u64* secs, const u32* bits, u32* isa, u64 n, u32* sa, u64* next, Build_Counts* counts);
// The others, once no end is tied: every suffix goes to its slot of sa. ends: the list of ends, `count` entries, as launch_split_followed gave it; isa is not the
// inverse array any more afterwards. updates: as below.
int launch_place_followed(csa_ctx* ctx, const u64* ends, u64 count, const u32* bits, u32* isa, u64 n, u32* sa, u64* updates);

// A list of groups of any size (heads, positions; *count_dev entries, at most `most`), group by group: how many of its entries are in small groups
// (counts->now_small) and where each tile's go; counts->next_small and counts->large are advanced by the two kinds. scratch: 2 words per
// RANK_TILE entries, for the call below.
int launch_count_by_size(csa_ctx* ctx, const u32* head, u64 most, const u64* count_dev, Build_Counts* counts, u32* scratch);
// Writes what was counted: small groups behind the entries that were at the front of next, large ones in front of those at its back; next
// holds cap entries.
int launch_split_by_size(csa_ctx* ctx, const u32* head, const u32* pos, u64 most, const u64* count_dev, u64* next, u64 cap, u32* scratch);
// counts->large_depth = how many symbols the suffixes of every group of the list share at least, as generation 0 leaves it (groups of one and the
// same key of key_bits bits, side by side).
int launch_large_depth(csa_ctx* ctx, const u64* list, u64 count, const u16* T, u64 n, const u32* code, int key_bits, Build_Counts* counts);
// Heads and positions of the entries of a list.
int launch_unpack_list(csa_ctx* ctx, const u64* list, u64 count, u32* head, u32* pos);

// The inverse array from sa (final slots) and the lists of tied suffixes. updates: n entries of scratch and 256 words.
int launch_make_inverse(csa_ctx* ctx, const u32* sa, u64 n, const u64* small_list, u64 small, const u64* large_list, u64 large, u32* isa, u64* updates);

// Children that did not fit a block's local sort (c: the counters read back, c.oversize > 0): sorted by (child, key) by the radix sort and
// ranked. The records are in `other`; the hole between the two ends of the list in front (n entries) takes the keys. The counters then
// stand as if the children had been sorted with the others, and launch_refine_by_text, which left the list alone, can be called again.
struct Oversize_Buffers
{
    void* sort_ws; size_t sort_bytes;       // csa_sort_workspace_bytes of the records
    u32* scratch;                           // oversize_scratch_bytes
    u8* work; size_t work_bytes;            // oversize_work_bytes
};
size_t oversize_scratch_bytes(u64 records);
size_t oversize_work_bytes(u64 records);
// The same carved from one piece of oversize_buffers_bytes, for up to `records` of them.
size_t oversize_buffers_bytes(u64 records);
Oversize_Buffers oversize_buffers(void* at, u64 records);
// An ordinary text has a few suffixes in a thousand in such children; a share of up to one in this many is room enough for them.
constexpr u64 OVERSIZE_SHARE = 64;
int sort_oversize_children(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& tab, const Build_Counts& c, u64 n, u64* front, u64* other, u32* sa, Build_Counts* counts,
                           const Oversize_Buffers& b);
