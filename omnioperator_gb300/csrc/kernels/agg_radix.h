// Radix aggregation: group-by with more groups than the hash partitions of the partitioned strategy
// can hold (agg_radix.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "plan.h"

namespace omg {

// A row's fine partition is bits [kRadixShift, kRadixShift + kRadixFineBits) of its key hash; a run
// uses the top `bits` of them.  The shared tables' index uses the hash's top 32 bits, the global table
// its low ones; a unit that is aggregated in several passes tells them apart by the bits below
// kRadixShift.
constexpr int kRadixFineBits = 14;
constexpr int kRadixFineParts = 1 << kRadixFineBits;
constexpr int kRadixShift = 18;
constexpr int kRadixMaxPassBits = 4;
constexpr int kRadixStepRows = 2048;  // rows that a CTA sorts and adds up at a time
constexpr int kRadixHllBits = 12;
constexpr int kRadixHllRegs = 1 << kRadixHllBits;

// A row as a record of 64-bit words: its input values (widest first, so that none straddles a
// word), then one byte per nullable input (1: NULL).
constexpr int kMaxRecWords = 12;
constexpr int kMaxRecSrc = 32;
struct RecSrc {
    int8_t input;
    int8_t width;  // bytes; 0: the input's NULL byte
    int8_t half;   // 16-byte values: word 0 or 1 of the value; else -1
    int8_t word;   // of the record
    int8_t shift;  // bits, within the word
};
struct RecLayout {
    int32_t words;
    int32_t nInputs;
    int32_t nSrc;
    int16_t off[kMaxInputs];      // byte offset of the value
    int16_t width[kMaxInputs];    // bytes of values of up to 8, else 0
    int16_t nullOff[kMaxInputs];  // byte offset of the NULL byte, -1: never NULL
    RecSrc src[kMaxRecSrc];       // by word
};

// The work of one CTA at a time: a partition's rows (it then holds all rows of its groups), or a
// run of them (multi).
struct RadixUnit {
    uint32_t first;  // record
    uint32_t rows;
    uint32_t multi;
    uint32_t pad;
};

struct RadixAgg {
    const uint64_t *records;
    const RadixUnit *units;
    int32_t nUnits;
    int32_t passBits;
    int32_t indexSize;
    int32_t pad;
    unsigned int *next;              // unit counter (zeroed)
    uint64_t *dense;                 // finished groups, slotWords words each
    unsigned long long *denseCount;  // (zeroed)
    uint64_t denseCap;
};

// Groups that a CTA's shared table holds, and the size of its index.
int32_t AggRadixSlots(int32_t smemStride, int32_t *indexSize);
// One pass over the keys of p's tiles: rows per fine partition, hist[kRadixFineParts], and HyperLogLog
// registers of the key hashes, regs[kRadixHllRegs] (both zeroed by the caller).
cudaError_t LaunchRadixKeys(const AggLaunch &p, unsigned int *hist, unsigned int *regs, cudaStream_t stream);
// The rows of p's tiles as records, grouped by partition; cursor[1 << bits] holds the partitions' first
// records.
cudaError_t LaunchRadixScatter(const AggLaunch &p, const RecLayout &l, int32_t bits, unsigned int *cursor,
    uint64_t *records, cudaStream_t stream);
// Aggregate the units.  Groups of whole partitions go to a.dense; p.table takes the groups of multi
// units, the special groups and those that found no shared slot (p.retry: record numbers).
cudaError_t LaunchRadixAgg(const AggLaunch &p, const RecLayout &l, const RadixAgg &a, uint64_t *spill,
    unsigned int *nSpill, uint32_t spillCap, cudaStream_t stream);
// The queued records (p.retryIn) and partial records (spillIn) into the grown p.table.
cudaError_t LaunchRadixRetry(const AggLaunch &p, const RecLayout &l, const uint64_t *records, uint64_t *spill,
    unsigned int *nSpill, uint32_t spillCap, const uint64_t *spillIn, uint32_t nSpillIn, int gridBlocks,
    cudaStream_t stream);

}  // namespace omg
