// Internal declarations of the build of a text that one block holds.
#pragma once
#include "common.cuh"

constexpr u64 TINY_BUILD_MAX = 16384;

struct Tiny_Result
{
    u64 status;             // the device status word
    u32 done;               // 0: nothing was written, the text is for the general build
    u32 tied;               // suffixes that shared a bin
    u32 partitions, max_partition;
};

// The suffix array of n <= TINY_BUILD_MAX symbols (16-byte aligned, padded) into sa40 (16-byte aligned). 1 << bucket_bits ranges of it are told apart for the
// count of partitions. result: pinned host memory, valid once the stream is synchronised.
int launch_tiny_build(csa_ctx* ctx, const u16* text, u64 n, u8* sa40, u32 p, int bucket_bits, Tiny_Result* result);
