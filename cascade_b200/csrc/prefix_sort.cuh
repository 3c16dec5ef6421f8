// Internal declarations of the resident build's generation 0: suffixes sorted by the first bits of their encoded symbols.
#pragma once
#include "batches.hpp"
#include "common.cuh"

// An order-preserving prefix code of the 16-bit symbols: entry s of a 65536-word table holds the symbol's code word in the top
// bits and its length (1 .. CODE_MAX_LEN) in the low 5 bits. Code words compare as their symbols do, so the bit strings of two
// suffixes compare as the suffixes do, and frequent symbols take few bits.
constexpr int CODE_MAX_LEN = 22;

// Groups of up to this many tied suffixes are ordered inside one block; larger ones go through the radix sort.
constexpr u32 SMALL_GROUP = 256;
constexpr u32 NARROW_GROUP = 15;
// What an entry of the suffix array holds while its suffix is still tied (no position: a resident build's n is below 2^32 - 2^26).
constexpr u32 SA_OPEN = 0xFFFFFFFFu;

// Counters that the kernels of a build leave for one another and for the host.
struct Build_Counts
{
    u32 small;          // entries of the list of small tied groups (filled from the front of its buffer)
    u32 large;          // entries of the list of large tied groups (filled from the back)
    u32 oversize;       // children that did not fit a block's local sort
    u32 oversize_records;
    u32 next_small;     // the same of the list being made
    u32 partitions;     // contiguous ranges of the suffix array, at most as many as asked for, that the first split's buckets form
    alignas(8) u32 batches;     // runs of children that the local sort takes
    u32 tries;          // and, beside it, blocks that have tried their first by even bins << 16 and those of them that have it still to order
    u32 crowded;        // and leaves to its second kernel: many of their records have the same key
    u32 medium;         // runs for its third
    u32 max_partition;  // suffixes of the largest partition
    u32 wide;           // not 0: a small group may have more than NARROW_GROUP members
    u32 now_small;      // entries that the last count by size found in small groups
    u32 large_depth;    // symbols that the suffixes of a large group share at least after the initial sort (launch_large_depth)
    u32 looked_at, lead_on, far_ties;       // what a sample of the small groups' entries says (launch_refine_by_text)
};
static_assert(sizeof(Build_Counts) <= (CSA_STATUS_WORD - CSA_COUNTS_WORD) * 8, "the counters lie before the status word");

struct Prefix_Sort
{
    u64 n;
    int b1, b2;             // bits of the first and the second split; b1 = 0: one split (or none) of b2 bits
    int key_bits;           // bits by which the suffixes end up sorted: b1 + 32, and up to FREE_BITS fewer where a parent has few children
    u32 parents, children;  // 1 << b1, 1 << b2
};

Prefix_Sort prefix_sort_plan(u64 n);
// Symbols that suffixes still tied after the sort share at least.
inline u64 shared_symbols(const Prefix_Sort& ps) { return u64((ps.key_bits - FREE_BITS) / CODE_MAX_LEN); }
// Device bytes of the tables (code, counts, offsets) beside the two record buffers of n 8-byte records.
size_t prefix_sort_table_bytes(const Prefix_Sort& ps);

struct Prefix_Tables
{
    u32* hist;          // 65536 symbol counts of the sample
    u32* code;          // 65536 entries of the code
    u32* cnt1;          // [parents] records by first digit
    u32* cur1;          // [parents] running places
    u32* par_off;       // [parents + 1] where each parent starts in the suffix array
    u32* tile0;         // [parents + 1] first tile of each parent in the second split
    u32* cnt2;          // [parents][children] records by second digit, then running places
    u32* child_off;     // [parents * children + 1] where each child starts in the suffix array
    uint4* batches;     // the local sort's batches (counts->batches of them): first slot, records, the run of children
    u32* over;          // children that did not fit a block, by their indices, from the front; runs of children left to the local sort's second kernel from the back
    u32* left;          // runs left to its third
};
bool prefix_sort_carve(Carver& cv, const Prefix_Sort& ps, Prefix_Tables& t);

// Orders the suffixes of T by the first key_bits bits of their encoding, up to FREE_BITS fewer where a parent has few children (shared_symbols). recA and recB: n records each. sa or, where that is null, sa40 (5-byte entries) receives every
// suffix that is alone with its key, at its final place, and SA_OPEN elsewhere; the tied ones go to `list` (the record buffer
// that is returned as *list; *records is the other one), small groups from the front, large ones from the back, as
// (first slot of the group << 32) | position, group by group. p only says how many partitions the statistics tell apart. Nothing is read back.
int launch_prefix_sort(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, u64* recA, u64* recB, u32* sa, u8* sa40, u32 p, Build_Counts* counts,
                       u64** list, u64** records, cudaEvent_t after_first_split);
// The records of the children that did not fit a block, as sort records: keys = (first slot of the child << 32) | key,
// vals = position.
int launch_pack_oversize(csa_ctx* ctx, const Prefix_Tables& t, u32 oversize, const u32* sa, u8* sa40);      // their slots, once sorted and ranked, as 5-byte entries
int launch_gather_oversize(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, u32 oversize, const u64* records, u64* keys, u32* vals, u32* cursor);

// The same for a text whose records do not all fit the device: one contiguous range of the suffix array at a time. The first split's
// buckets are counted once (cnt1, 1 << b1 of them); a part is a run of buckets with `size` suffixes in all, for which the text is
// encoded again. There are always two splits.
Prefix_Sort prefix_sort_part_plan(u64 n);
int launch_prefix_counts(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, Build_Counts* counts);
// recA, recB, sa: `size` entries each; slots count from the part's first. The list of tied suffixes is left in recA.
int launch_prefix_sort_part(csa_ctx* ctx, const Prefix_Sort& ps, const Prefix_Tables& t, const u16* T, u32 first_bin, u32 bins, u64 size, u64* recA, u64* recB, u32* sa,
                            Build_Counts* counts);
