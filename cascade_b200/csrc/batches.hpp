// Which runs of children the resident build's local sort takes at once. Plain C++: the kernel that forms the batches and the host code that makes room for their list go by the same rules.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CSA_BOTH __host__ __device__ __forceinline__
#else
#define CSA_BOTH inline
#endif

constexpr uint32_t SORT_BLOCK = 256, SORT_ITEMS = 16, SORT_CAP = SORT_BLOCK * SORT_ITEMS, SORT_MOST = SORT_CAP - 4;      // records of the largest batch
constexpr int FREE_BITS = 4;                // of a key in a batch take its slot's last bits. A run of children has that many fewer bits than all of a parent's, or, where a parent has few children, up to
constexpr uint32_t FEW_CHILDREN = 4;        // so many, and the key's last bits are not looked at: what they told apart is left to the ties
constexpr uint32_t SEGMENT = 64, SHORT_SEGMENT = 8;     // children whose batches one thread forms: they end with a segment
constexpr uint32_t SHORT_BATCH = 1024;      // records of a batch of a text of one split, so that it has one for every SM

// Children of the longest run that is one batch, where a parent has `children`.
CSA_BOTH uint32_t longest_run(const uint32_t children)
{
    const uint32_t few = children < FEW_CHILDREN ? children : FEW_CHILDREN, part = children >> FREE_BITS;
    return part > few ? part : few;
}

// The child behind the batch that begins with child i: it ends with a segment, with the longest run, or before a child with which it would have more than `most` records; it has one child at least.
// off[0 .. children]: where the children of the parent start, and its end.
CSA_BOTH uint32_t batch_end(const uint32_t* const off, const uint32_t i, const uint32_t children, const uint32_t segment, const uint32_t most)
{
    const uint32_t run = i + longest_run(children), stop = (i / segment + 1) * segment;
    uint32_t a = i + 1, b = (run < stop ? run : stop) + 1;
    if(b > children + 1) b = children + 1;
    while(b - a > 1)
    {
        const uint32_t m = (a + b) >> 1;
        if(off[m] - off[i] <= most) a = m; else b = m;
    }
    return a;
}

// Entries of the list of batches: each has a child that no other has. Not fewer: runs of nearly empty children end by their number, so no count of records bounds them (2.2e6 symbols over 2048 children of
// which every other one holds nearly everything: 1210 batches; 2 n / SORT_MOST and the segments' ends would be 1139). 16 bytes a child of some 1500 suffixes.
CSA_BOTH uint64_t most_batches(const uint32_t parents, const uint32_t children) { return uint64_t(parents) * children; }
