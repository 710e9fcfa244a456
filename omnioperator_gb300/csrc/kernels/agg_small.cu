// A whole small aggregation in one launch.
//
// A call of some thousand rows is its fixed costs: a table initialised, aggregated, counted and extracted
// in launches of their own, each with its allocations, and waits between them.  Here one CTA reads the
// batches (over the CPU-GPU link when they are the host's), aggregates them in shared memory and
// writes the groups to the output columns and their number to pinned memory: one launch, one wait, and
// no device memory but a device caller's outputs.
#include <cstdint>
#include <cuda_runtime.h>

#include "agg_device.cuh"
#include "agg_extract.cuh"
#include "agg_small.h"
#include "agg_steps.cuh"
#include "launch.h"

namespace omg {
namespace {

static_assert(kSmallStepRows == kStepRows, "a step of the launch is a step of the table");
constexpr size_t kSmallSmemBytes = 208 * 1024;

// Rows row0 and up of a batch.
struct SmallRows {
    const BatchDesc &b;
    const int16_t *width;
    int64_t row0;
    __device__ __forceinline__ const char *RowAt(int input, int w, uint32_t r) const
    {
        return static_cast<const char *>(b.cols[input]) + (row0 + r) * w;
    }
    __device__ __forceinline__ int Width(int input) const { return width[input]; }
    __device__ __forceinline__ bool Nullable(int input) const { return b.nulls[input] != nullptr; }
    __device__ __forceinline__ uint32_t NullByte(int input, uint32_t r) const
    {
        return __ldg(reinterpret_cast<const unsigned char *>(b.nulls[input]) + ((row0 + r) >> 3));
    }
    __device__ __forceinline__ uint32_t NullBit(uint32_t byte, uint32_t r) const { return (byte >> ((row0 + r) & 7)) & 1u; }
};

template <int kKind>
__global__ void __launch_bounds__(kStepThreads, 1) AggSmallKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ AggExtract e, const __grid_constant__ SmallArgs a)
{
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ BatchDesc batches[kSmallMaxSteps];
    __shared__ unsigned int used;
    __shared__ unsigned int missed;
    __shared__ unsigned int warpSums[kStepThreads / 32];
    const int sw = p.smemStride;
    const int kw = p.table.keyWords;
    const unsigned int nSlots = static_cast<unsigned int>(p.smemSlots);
    const int nAll = static_cast<int>(nSlots) + kSpecialSlots;
    const StepTable tab = MakeStepTable(smem, nAll, sw, kw, nSlots, a.indexSize, &used, warpSums);
    {
        const uint64_t *from = reinterpret_cast<const uint64_t *>(a.batches);
        uint64_t *to = reinterpret_cast<uint64_t *>(batches);
        for (int i = threadIdx.x; i < a.nBatches * static_cast<int>(sizeof(BatchDesc) / 8); i += kStepThreads) {
            to[i] = from[i];
        }
    }
    InitStepTable(p, tab);
    if (threadIdx.x == 0) {
        missed = 0;
    }
    __syncthreads();
    for (int i = 0; i < a.nSteps; ++i) {
        const SmallStep step = a.steps[i];
        AggregateStep<kKind>(p, SmallRows{batches[step.batch], a.width, step.row0}, static_cast<uint32_t>(step.rows), tab,
            [](const RowKey &) { return true; }, [&](uint32_t, const RowKey &) { missed = 1; });
    }
    if (missed != 0) {
        if (threadIdx.x == 0) {
            a.result[3] = 1;
        }
        return;
    }
    // The groups out: the special ones, if they have rows, behind the others.
    const unsigned int groups = min(used, nSlots);
    const bool isNull = tab.st[p.accs[0].word] != 0;
    const bool isEmpty = tab.st[sw + p.accs[0].word] != 0;
    const unsigned int rows = groups + (isNull ? 1 : 0) + (isEmpty ? 1 : 0);
    for (int o = 0; o < e.nOut; ++o) {
        for (unsigned int i = threadIdx.x; i < (rows + 31) / 32; i += kStepThreads) {
            reinterpret_cast<unsigned int *>(e.out[o].nulls)[i] = 0;
        }
    }
    __threadfence_system();  // the bitmaps may be host memory: cleared before any bit is set
    __syncthreads();
    AggTable t;
    t.slots = smem;
    t.capacity = static_cast<uint64_t>(nAll);
    t.slotWords = sw;
    t.keyWords = kw;
    t.specialUsed = nullptr;
    t.groupCount = nullptr;
    for (unsigned int i = threadIdx.x; i < rows; i += kStepThreads) {
        uint64_t s = i + kSpecialSlots;
        const uint64_t *slot = smem + s * sw;
        if (i >= groups) {
            const int special = i == groups && isNull ? kNullSlotOffset : kSentinelSlotOffset;
            s = t.capacity + special;
            slot = smem + static_cast<int64_t>(special) * sw;
        }
        WriteGroup(e, t, s, slot, i);
    }
    if (threadIdx.x == 0) {
        a.result[0] = rows;
    }
}

}  // namespace

int32_t AggSmallSlots(int32_t smemStride, int32_t *indexSize)
{
    return StepTableSlots(smemStride, kSmallSmemBytes, indexSize);
}

cudaError_t LaunchAggSmall(const AggLaunch &p, const AggExtract &e, const SmallArgs &a, cudaStream_t stream)
{
    auto kernel = p.key.kind == KEY_SINGLE ? AggSmallKernel<KEY_SINGLE> : AggSmallKernel<KEY_PACKED>;
    const cudaError_t err = EnsureDynamicSmem(reinterpret_cast<const void *>(kernel), kSmallSmemBytes);
    if (err != cudaSuccess) {
        return err;
    }
    kernel<<<1, kStepThreads, kSmallSmemBytes, stream>>>(p, e, a);
    return cudaGetLastError();
}

}  // namespace omg
