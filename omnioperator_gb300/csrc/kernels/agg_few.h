// Group-by with a handful of groups (agg_few.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "plan.h"

namespace omg {

// Where the threads' private states are in a CTA's shared memory: accumulator a's state of group g of
// thread t is element g * kFewThreads + t from byte off[a] (two planes for an exact sum: positive, then
// negative magnitudes, planeStep bytes apart).  off[a] < 0: the accumulator keeps no state (NULLS of an
// input without NULLs).
constexpr int kFewThreads = 256;
struct FewLayout {
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

// The layout for p's accumulators; nullable: bit i: input i has NULLs.  False: an accumulator without a
// private form, or no room for four groups.
bool LayoutAggFew(const AggLaunch &p, uint32_t nullable, FewLayout *l);
int LaunchAggFewGrid();
cudaError_t LaunchAggFew(const AggLaunch &p, const FewLayout &l, uint64_t *spill, unsigned int *nSpill,
    uint32_t spillCap, cudaStream_t stream);

}  // namespace omg
