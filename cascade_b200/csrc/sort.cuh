// Internal declarations shared by the translation units of the device library.
#pragma once
#include "common.cuh"

// Drops the digit-pass events collected for the context's device.
void sort_reset_timing(csa_ctx* ctx);
// Frees the context's digit-pass timer.
void sort_free_timing(csa_ctx* ctx);

// Device address of the digit histograms ([pass][256] 64-bit counts) left in the workspace by the last csa_sort_pairs of n records.
const u64* sort_workspace_histograms(void* workspace, size_t workspace_bytes, u64 n);

// Test hook of the part-at-a-time build: the offset added to every position that is put into a lane.
void stream_set_position_offset(u64 offset);

// Sorts the segments [seg_off_host[s], seg_off_host[s + 1]) of one record array, each on its own, in one set of launches and
// without a read-back; every pass runs, so the records end in the alt buffers iff the number of passes is odd. Values are
// 32-bit (or absent: both pointers null). Every segment holds fewer than 2^30 records.
size_t sort_segments_workspace_bytes(u64 n, u32 segs);
int sort_segments(csa_ctx* ctx, u64* keys, u64* keys_alt, u32* vals, u32* vals_alt, const u64* seg_off_host, u32 segs, int begin_bit, int end_bit, void* workspace,
                  size_t workspace_bytes, int* in_alt);

// Buckets by the top bits of evenly spread keys, each finished inside one block (bucket_sort.cu).
constexpr int BUCKET_MAX_BITS = 15;                 // a block counts them in shared memory
constexpr u64 BUCKET_MAX_RECORDS = 8192;            // what a block holds
constexpr u64 BUCKET_MAX_TOTAL = u64(1) << 26;      // records of a sort by buckets: 2048 a bucket
// Top bits by which n records are split into buckets of 512 to 2048 on average.
int bucket_sort_bits(u64 n);
// What the counts say, on the device; zeroed before.
struct Bucket_Findings
{
    u64 differ;         // bits in which keys differ
    u32 uneven;         // a bucket does not fit a block, or digit passes would skip so many digits that they are the faster way
    u32 left;           // buckets that turned out to be uneven inside
};
// The buckets' starts (1 << bits of them, and the end; zeroed before), the digit offsets of the passes by the lower low_bits of the bucket number and
// by the others, and the verdict: `found`, and in *verdict (pinned host memory, once the stream has been waited for) the size of the largest bucket or 0
// for uneven keys. Queued. least_digits: digits of 8 bits from begin_bit on in which the keys have to differ.
int launch_bucket_plan(csa_ctx* ctx, const u64* keys, u64 n, int begin_bit, int end_bit, int bits, int low_bits, int least_digits, u32* starts, u64* low_base, u64* high_base,
                       Bucket_Findings* found, u64* verdict);
// Every bucket (starts == nullptr: all n records) sorted by the key bits [begin_bit, top), stably; largest: no bucket holds more. found->left is counted up.
int launch_bucket_sort(csa_ctx* ctx, const u64* kin, u64* kout, const void* vin, void* vout, u32 val_bytes, const u32* starts, u32 buckets, u64 n, u64 largest, Bucket_Findings* found,
                       int begin_bit, int top);
