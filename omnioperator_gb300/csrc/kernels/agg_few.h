// Group-by with a handful of groups (agg_few.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "plan.h"

namespace omg {

// Where the threads' private states are in a CTA's shared memory: accumulator a's state of group g of
// thread t is element g * threads + t from byte off[a] (two planes, planeStep bytes apart, for an exact sum:
// positive, then negative magnitudes, and for a sum of doubles: the sum, then its rounding errors).  off[a] < 0:
// the accumulator keeps no state (NULLS of an input without NULLs).
constexpr int kFewMaxThreads = 256;
constexpr int kFewMinThreads = 128;  // in steps of 64
struct FewLayout {
    int32_t threads;     // of a CTA
    int32_t maxGroups;   // with private states
    int32_t firstSlot;   // the first slot with private states: 0 when the key may be NULL, else 2
    int32_t smemBytes;
    int32_t off[kMaxAccs];
    int32_t planeStep[kMaxAccs];
    // The accumulators with a state, but COUNT_ALL, by input: those of input[i] (values of width[i] bytes)
    // are acc[firstAcc[i]] to acc[firstAcc[i + 1] - 1].
    int32_t nInputs;
    int16_t input[kMaxInputs];
    int16_t width[kMaxInputs];
    int16_t firstAcc[kMaxInputs + 1];
    int16_t acc[kMaxAccs];
};

// The layout for p's accumulators and `slots` groups, the special ones among them; nullable: bit i: input i has
// NULLs.  False: an accumulator without a private form, or no room for them, or for four groups.
bool LayoutAggFew(const AggLaunch &p, uint32_t nullable, uint64_t slots, FewLayout *l);
int LaunchAggFewGrid();
cudaError_t LaunchAggFew(const AggLaunch &p, const FewLayout &l, uint64_t *spill, unsigned int *nSpill,
    uint32_t spillCap, cudaStream_t stream);

}  // namespace omg
