// A whole small aggregation in one launch (agg_small.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "plan.h"

namespace omg {

constexpr int kSmallMaxSteps = 8;
constexpr int kSmallStepRows = 2048;
struct SmallStep {
    int32_t batch;
    int32_t row0;
    int32_t rows;  // at most kSmallStepRows
    int32_t pad;
};
// result (memory that the host reads): [0] rows written, [1] an overflow is an error, [2] groups whose overflow
// depends on the row order, [3] more groups than slots (nothing written), [4] kernel error.  Zeroed by the
// caller.
struct SmallArgs {
    const BatchDesc *batches;  // read once (may be pinned host memory)
    int32_t nBatches;          // at most kSmallMaxSteps
    int32_t nSteps;
    SmallStep steps[kSmallMaxSteps];
    int16_t width[kMaxInputs];  // of inputs of up to 8 bytes, else 0
    int32_t indexSize;
    int32_t pad;
    unsigned long long *result;
};

// Groups that the launch can hold, and the size of its index.
int32_t AggSmallSlots(int32_t smemStride, int32_t *indexSize);
// p: key, accumulators, table.slotWords / keyWords, smemSlots; e: outputs (their NULL bitmaps need not be
// cleared), error and nAmbiguous.
cudaError_t LaunchAggSmall(const AggLaunch &p, const AggExtract &e, const SmallArgs &a, cudaStream_t stream);

}  // namespace omg
