// Radix aggregation for many groups.
//
// With more groups than fit the shared tables of a few partitions, every row used to update a global
// table: a random slot of hundreds of megabytes, 6-10 atomics per row, the atomics of a hot key all on
// one address, and a table sized from a 65,536-row sample whose undersized probe chains cost
// 300 instructions a row.  Here one pass over the keys counts rows per fine hash partition and
// distinct keys (HyperLogLog), a scatter pass turns the rows into records grouped by as many
// partitions as the distinct keys need, and a CTA aggregates a partition at a time in a shared table.
// A partition is all rows of its groups, so its table is final: it is appended to a dense array of
// groups that no hash table holds.  A partition with a hot key is cut into units whose tables are
// merged into the (small) global table.
#include <cstdint>
#include <cuda_runtime.h>

#include "agg_device.cuh"
#include "agg_radix.h"
#include "agg_steps.cuh"
#include "device_common.cuh"
#include "launch.h"

namespace omg {
namespace {

// A row's inputs in its record.
struct RecRow {
    const RecLayout &l;
    const char *rec;
    __device__ __forceinline__ bool Null(int input) const { return l.nullOff[input] >= 0 && __ldg(rec + l.nullOff[input]) != 0; }
    __device__ __forceinline__ uint64_t Bits(int input, int width) const { return LoadBitsRO(rec + l.off[input], 0, width); }
    __device__ __forceinline__ const uint64_t *Wide(int input) const
    {
        return reinterpret_cast<const uint64_t *>(rec + l.off[input]);
    }
};

__device__ __forceinline__ const char *RecAt(const RecLayout &l, const uint64_t *records, uint64_t i)
{
    return reinterpret_cast<const char *>(records + i * l.words);
}

__device__ __forceinline__ unsigned int FinePart(uint64_t hash)
{
    return static_cast<unsigned int>(hash >> kRadixShift) & (kRadixFineParts - 1);
}

// The records of a step.
struct RecRows {
    const RecLayout &l;
    const char *step;  // the first
    __device__ __forceinline__ const char *RowAt(int input, int, uint32_t r) const
    {
        return step + r * (static_cast<uint32_t>(l.words) * 8u) + l.off[input];
    }
    __device__ __forceinline__ int Width(int input) const { return l.width[input]; }
    __device__ __forceinline__ bool Nullable(int input) const { return l.nullOff[input] >= 0; }
    __device__ __forceinline__ uint32_t NullByte(int input, uint32_t r) const
    {
        return __ldg(reinterpret_cast<const unsigned char *>(
            step + r * (static_cast<uint32_t>(l.words) * 8u) + l.nullOff[input]));
    }
    __device__ __forceinline__ uint32_t NullBit(uint32_t byte, uint32_t) const { return byte != 0 ? 1u : 0u; }
};

// ------------------------------------------------------------------ key pass
constexpr int kKeyThreads = 512;
constexpr int kKeyRows = 4;  // rows per thread whose key loads are in flight together
constexpr size_t kKeySmem = sizeof(unsigned int) * (kRadixFineParts + kRadixHllRegs);

template <int kKind>
__global__ void __launch_bounds__(kKeyThreads, 2) RadixKeyKernel(const __grid_constant__ AggLaunch p, unsigned int *hist,
    unsigned int *regs)
{
    extern __shared__ __align__(16) uint64_t smem[];
    unsigned int *h = reinterpret_cast<unsigned int *>(smem);
    unsigned int *r = h + kRadixFineParts;
    for (int i = threadIdx.x; i < kRadixFineParts + kRadixHllRegs; i += kKeyThreads) {
        h[i] = 0;
    }
    __syncthreads();
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        const TileDesc tile = p.tiles[t];
        const BatchDesc &b = p.batches[tile.batch];
        for (int r0 = threadIdx.x; r0 < tile.rows; r0 += kKeyRows * kKeyThreads) {
            uint32_t use = 0;
#pragma unroll
            for (int j = 0; j < kKeyRows; ++j) {
                use |= r0 + j * kKeyThreads < tile.rows ? 1u << j : 0u;
            }
            RowKey k[kKeyRows];
            ReadKeys<kKind, kKeyRows>(p.key, BatchRows<kKeyThreads>{b, static_cast<int64_t>(tile.row0) + r0}, use, k);
#pragma unroll
            for (int j = 0; j < kKeyRows; ++j) {
                if (((use >> j) & 1u) == 0) {
                    continue;
                }
                atomicAdd(&h[FinePart(k[j].hash)], 1u);
                if (k[j].special < 0) {
                    const unsigned int reg = static_cast<unsigned int>(k[j].hash) & (kRadixHllRegs - 1);
                    const unsigned int rank = static_cast<unsigned int>(
                        __clzll(static_cast<long long>(k[j].hash | (1ull << kRadixHllBits))) + 1);
                    if (rank > *reinterpret_cast<volatile unsigned int *>(&r[reg])) {
                        atomicMax(&r[reg], rank);
                    }
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRadixFineParts; i += kKeyThreads) {
        if (h[i] != 0) {
            atomicAdd(&hist[i], h[i]);
        }
    }
    for (int i = threadIdx.x; i < kRadixHllRegs; i += kKeyThreads) {
        if (r[i] != 0) {
            atomicMax(&regs[i], r[i]);
        }
    }
}

// ------------------------------------------------------------------ scatter
// Four tiles per step: each row takes its rank within (step, partition) from a shared counter, the
// step reserves each partition's records with one global atomic, and a row is written as one record.
// What bounds the pass is the number of store requests to distinct lines, 38 G/s whatever the number of
// partitions from 64 up and whatever their width (2^26 records of 32 bytes: 3.45 ms as two 16-byte
// stores each, 1.75 ms as one of 32 bytes), so records of three or more words are padded to 32 bytes and
// stored 32 bytes at a time; columns apart would take a request each.  Every pass over rows loads several
// rows' values before it uses any, and what must outlive a pass is in shared memory: a register spill is a
// store request too (packed keys spill 24 bytes a thread at 64 registers, and none at the 128 that were
// slower).  Wide records are bound by latency before that: 32 warps of 64 registers with three
// sources in flight instead of 16 of 128 with six took 2^26 records of a two-column key from 3.10 to 2.35 ms
// (two sources 2.69; 2^24 of 16 bytes 0.44 -> 0.36; steps of eight tiles 2.42 and 0.41).
constexpr int kScatterThreads = 1024;
constexpr int kScatterTiles = 4;
constexpr int kTileThreadRows = kTileRows / kScatterThreads;
constexpr int kScatterRows = kScatterTiles * kTileRows;
constexpr unsigned int kNoPart = 0xffffffffu;

constexpr int kMoveRows = 2;  // rows whose loads are in flight together

// Words w to w + 3 of the rows' records; v starts over.
__device__ __forceinline__ void StoreWords(const RecLayout &l, int w, uint32_t use, uint64_t *const (&dst)[kMoveRows],
    uint64_t (&v)[4][kMoveRows])
{
#pragma unroll
    for (int j = 0; j < kMoveRows; ++j) {
        if ((use >> j) & 1u) {
            if (l.words >= 4) {
                asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(dst[j] + w), "l"(v[0][j]), "l"(v[1][j]),
                    "l"(v[2][j]), "l"(v[3][j])
                    : "memory");
            } else if (l.words == 2) {
                *reinterpret_cast<ulonglong2 *>(dst[j]) = make_ulonglong2(v[0][j], v[1][j]);
            } else {
                dst[j][0] = v[0][j];
            }
        }
        v[0][j] = v[1][j] = v[2][j] = v[3][j] = 0;
    }
}

// The values that rows row0 + j * kScatterThreads (bit j of `use`) put into sources [s0, s0 + kSrcBatch).
constexpr int kSrcBatch = 3;

__device__ __forceinline__ void LoadSources(const RecLayout &l, int s0, const BatchDesc &b, int64_t row0, uint32_t use,
    uint64_t (&x)[kSrcBatch][kMoveRows])
{
#pragma unroll
    for (int k = 0; k < kSrcBatch; ++k) {
        if (s0 + k >= l.nSrc) {
            break;
        }
        const RecSrc s = l.src[s0 + k];
        if (s.width == 0) {
            const unsigned char *nulls = reinterpret_cast<const unsigned char *>(b.nulls[s.input]);
            LoadBitsRows<kMoveRows>(
                [&](int j) { return reinterpret_cast<const char *>(nulls) + ((row0 + j * kScatterThreads) >> 3); }, 1,
                nulls != nullptr ? use : 0u, x[k]);
        } else {
            const char *col = static_cast<const char *>(b.cols[s.input]) + (s.half > 0 ? 8 : 0);
            const int stride = s.half >= 0 ? 16 : s.width;
            LoadBitsRows<kMoveRows>([&](int j) { return col + (row0 + j * kScatterThreads) * stride; }, s.width, use,
                x[k]);
        }
    }
}

template <int kKind>
__global__ void __launch_bounds__(kScatterThreads, 1) RadixScatterKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ RecLayout l, int32_t bits, unsigned int *cursor, uint64_t *records)
{
    // Rows of the step per partition, then the partitions' first records; each row's partition << 16 | rank
    // (both at most 2^14).
    extern __shared__ __align__(16) uint64_t smem[];
    const int nParts = 1 << bits;
    unsigned int *at = reinterpret_cast<unsigned int *>(smem);
    unsigned int *cnt = at + kScatterRows;
    for (int t0 = blockIdx.x * kScatterTiles; t0 < p.nTiles; t0 += gridDim.x * kScatterTiles) {
        for (int i = threadIdx.x; i < nParts; i += kScatterThreads) {
            cnt[i] = 0;
        }
        __syncthreads();
        const int nTiles = min(kScatterTiles, p.nTiles - t0);
#pragma unroll 1
        for (int g = 0; g < nTiles * kTileThreadRows; g += kMoveRows) {
            const TileDesc tile = p.tiles[t0 + g / kTileThreadRows];
            const int r0 = g % kTileThreadRows * kScatterThreads + threadIdx.x;
            uint32_t use = 0;
#pragma unroll
            for (int j = 0; j < kMoveRows; ++j) {
                use |= r0 + j * kScatterThreads < tile.rows ? 1u << j : 0u;
            }
            RowKey k[kMoveRows];
            ReadKeys<kKind, kMoveRows>(p.key,
                BatchRows<kScatterThreads>{p.batches[tile.batch], static_cast<int64_t>(tile.row0) + r0}, use, k);
#pragma unroll
            for (int j = 0; j < kMoveRows; ++j) {
                unsigned int a = kNoPart;
                if ((use >> j) & 1u) {
                    const unsigned int q = FinePart(k[j].hash) >> (kRadixFineBits - bits);
                    a = (q << 16) | atomicAdd(&cnt[q], 1u);
                }
                at[(g + j) * kScatterThreads + threadIdx.x] = a;
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int i = threadIdx.x; i < nParts; i += kScatterThreads) {
            const unsigned int c = cnt[i];
            if (c != 0) {
                cnt[i] = atomicAdd(&cursor[i], c);
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int g = 0; g < nTiles * kTileThreadRows; g += kMoveRows) {
            const TileDesc tile = p.tiles[t0 + g / kTileThreadRows];
            const BatchDesc &b = p.batches[tile.batch];
            const int64_t row0 = static_cast<int64_t>(tile.row0) + g % kTileThreadRows * kScatterThreads + threadIdx.x;
            uint64_t *dst[kMoveRows];
            uint32_t use = 0;
#pragma unroll
            for (int j = 0; j < kMoveRows; ++j) {
                const unsigned int a = at[(g + j) * kScatterThreads + threadIdx.x];
                use |= a != kNoPart ? 1u << j : 0u;
                dst[j] = a != kNoPart ? records + static_cast<uint64_t>(cnt[a >> 16] + (a & 0xffffu)) * l.words : nullptr;
            }
            // Sources are in word order; a batch of them is loaded, then put into its words.
            uint64_t v[4][kMoveRows];  // words w to w + 3, w a multiple of 4
#pragma unroll
            for (int j = 0; j < kMoveRows; ++j) {
                v[0][j] = v[1][j] = v[2][j] = v[3][j] = 0;
            }
            int w = 0;
            for (int s0 = 0; s0 < l.nSrc; s0 += kSrcBatch) {
                uint64_t x[kSrcBatch][kMoveRows];
                LoadSources(l, s0, b, row0, use, x);
#pragma unroll
                for (int k = 0; k < kSrcBatch; ++k) {
                    if (s0 + k >= l.nSrc) {
                        break;
                    }
                    const RecSrc s = l.src[s0 + k];
                    if ((s.word & ~3) != w) {
                        StoreWords(l, w, use, dst, v);
                        w = s.word & ~3;
                    }
#pragma unroll
                    for (int j = 0; j < kMoveRows; ++j) {
                        uint64_t y = x[k][j];
                        if (s.width == 0) {
                            y = (y >> ((row0 + j * kScatterThreads) & 7)) & 1u;
                        }
                        y <<= s.shift;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            v[i][j] |= (s.word & 3) == i ? y : 0ull;
                        }
                    }
                }
            }
            StoreWords(l, w, use, dst, v);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ aggregation
constexpr size_t kRadixSmemBytes = 112 * 1024;  // two CTAs per SM

// The generic path of one record: straight into the global table, or queued.
__device__ __noinline__ void GlobalRecord(const AggLaunch &p, const RecLayout &l, const uint64_t *records, uint64_t i,
    RowKey key, int kind, unsigned int *newGroups)
{
    bool inserted = false;
    const int64_t g = GlobalFind(p.table, p.key, key, p.maxProbe, p.error, &inserted, p.waitBudget, kind);
    if (g < 0) {
        QueueRetry(p, 0, static_cast<int64_t>(i));
        return;
    }
    if (inserted) {
        atomicAdd(newGroups, 1u);
    }
    // The record as row 0 of a batch of its own.
    const char *rec = RecAt(l, records, i);
    BatchDesc b;
    for (int c = 0; c < l.nInputs; ++c) {
        b.cols[c] = rec + l.off[c];
        b.nulls[c] = l.nullOff[c] >= 0 ? reinterpret_cast<const uint8_t *>(rec + l.nullOff[c]) : nullptr;
        b.offs[c] = nullptr;
    }
    b.rows = 1;
    b.rowBase = 0;
    RowIn in;
    in.k = key;
    in.nulls = 0;
    for (int r = 0; r < kRegInputs; ++r) {
        in.v[r] = 0;
        if (r < p.nRegInputs) {
            const int c = p.regInput[r];
            in.v[r] = LoadBitsRO(b.cols[c], 0, p.regWidth[r]);
            in.nulls |= (NullRO(b.nulls[c], 0) ? 1u : 0u) << r;
        }
    }
    UpdateStates(p, b, 0, in, p.table.slots + g * p.table.slotWords + p.table.keyWords);
}

static_assert(kStepRows == kRadixStepRows, "units are whole steps");

template <int kKind>
__global__ void __launch_bounds__(kStepThreads, 2) RadixAggKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ RecLayout l, const __grid_constant__ RadixAgg a, const __grid_constant__ SpillArgs sp)
{
    // The slots (the special ones first), the step's rows in slot order, the exchange buffers, the index, the
    // counters.
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ unsigned int newGroups;
    __shared__ unsigned int unitIndex;
    __shared__ unsigned int used;
    __shared__ unsigned int warpSums[kStepThreads / 32];
    __shared__ unsigned long long denseBase;
    const int sw = p.table.slotWords;
    const int ss = p.smemStride;
    const int kw = p.table.keyWords;
    const unsigned int nSlots = static_cast<unsigned int>(p.smemSlots);
    const int nAll = static_cast<int>(nSlots) + kSpecialSlots;
    const StepTable tab = MakeStepTable(smem, nAll, ss, kw, nSlots, a.indexSize, &used, warpSums);
    InitStepTable(p, tab);
    if (threadIdx.x == 0) {
        newGroups = 0;
    }
    const unsigned int passMask = (1u << a.passBits) - 1u;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            unitIndex = atomicAdd(a.next, 1u);
        }
        __syncthreads();
        if (unitIndex >= static_cast<unsigned int>(a.nUnits)) {
            break;
        }
        const RadixUnit unit = a.units[unitIndex];
        const uint32_t steps = (unit.rows + kStepRows - 1) / kStepRows;
        const uint32_t stepRows = (unit.rows + steps - 1) / steps;
        for (unsigned int pass = 0; pass <= passMask; ++pass) {
            for (uint32_t r0 = 0; r0 < unit.rows; r0 += stepRows) {
                AggregateStep<kKind>(p, RecRows{l, RecAt(l, a.records, static_cast<uint64_t>(unit.first) + r0)},
                    min(stepRows, unit.rows - r0), tab,
                    [&](const RowKey &k) {
                        return k.special >= 0 ? pass == 0
                                              : ((k.hash >> (kRadixShift - kRadixMaxPassBits)) & passMask) == pass;
                    },
                    [&](uint32_t r, const RowKey &k) {
                        GlobalRecord(p, l, a.records, static_cast<uint64_t>(unit.first) + r0 + r, k, kKind, &newGroups);
                    });
            }
            const unsigned int groups = min(used, nSlots);
            if (threadIdx.x < kSpecialSlots) {
                const int s = threadIdx.x;
                uint64_t *slot = smem + static_cast<int64_t>(s) * ss;
                if (slot[kw + p.accs[0].word] != 0) {
                    atomicExch(&p.table.specialUsed[s], 1u);
                    MergeStates(p, p.accs, p.nAccs, slot + kw, p.table.slots + (p.table.capacity + s) * sw + kw);
                    InitSlot(p, slot);
                }
            }
            uint64_t *first = smem + static_cast<int64_t>(kSpecialSlots) * ss;
            if (unit.multi != 0) {
                for (unsigned int i = threadIdx.x; i < groups; i += kStepThreads) {
                    MergeRecord<kKind>(p, sp, first + static_cast<int64_t>(i) * ss, &newGroups);
                }
            } else {
                // A whole partition: append its groups.
                if (threadIdx.x == 0) {
                    denseBase = atomicAdd(a.denseCount, static_cast<unsigned long long>(groups));
                }
                __syncthreads();
                if (denseBase + groups > a.denseCap) {
                    SetError(p.error, 4);  // the host sized it for every slot of every pass, so this is a bug
                } else {
                    uint64_t *dst = a.dense + denseBase * sw;
                    for (unsigned int w = threadIdx.x; w < groups * sw; w += kStepThreads) {
                        const unsigned int g = w / sw;
                        dst[w] = first[g * ss + (w - g * sw)];
                    }
                }
            }
            __syncthreads();
            for (unsigned int i = threadIdx.x; i < groups; i += kStepThreads) {
                InitSlot(p, first + static_cast<int64_t>(i) * ss);
            }
            for (int i = threadIdx.x; i < a.indexSize; i += kStepThreads) {
                tab.index[i] = 0;
            }
            if (threadIdx.x == 0) {
                used = 0;
            }
            __syncthreads();
        }
    }
    if (threadIdx.x == 0 && newGroups != 0) {
        atomicAdd(p.table.groupCount, static_cast<unsigned long long>(newGroups));
    }
}

template <int kKind>
__global__ void __launch_bounds__(512) RadixRetryKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ RecLayout l, const uint64_t *records, const __grid_constant__ SpillArgs sp)
{
    __shared__ unsigned int newGroups;
    if (threadIdx.x == 0) {
        newGroups = 0;
    }
    __syncthreads();
    const int64_t gtid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = gtid; i < p.nRetryIn; i += stride) {
        const uint64_t r = p.retryIn[i] & 0xffffffffull;
        const RowKey key = ReadKeyOf(p.key, RecRow{l, RecAt(l, records, r)}, kKind);
        GlobalRecord(p, l, records, r, key, kKind, &newGroups);
    }
    for (int64_t i = gtid; i < sp.nSpillIn; i += stride) {
        MergeRecord<kKind>(p, sp, sp.spillIn + i * p.table.slotWords, &newGroups);
    }
    __syncthreads();
    if (threadIdx.x == 0 && newGroups != 0) {
        atomicAdd(p.table.groupCount, static_cast<unsigned long long>(newGroups));
    }
}

}  // namespace

int32_t AggRadixSlots(int32_t smemStride, int32_t *indexSize)
{
    return StepTableSlots(smemStride, kRadixSmemBytes, indexSize);
}

cudaError_t LaunchRadixKeys(const AggLaunch &p, unsigned int *hist, unsigned int *regs, cudaStream_t stream)
{
    if (p.nTiles <= 0) {
        return cudaSuccess;
    }
    auto kernel = p.key.kind == KEY_SINGLE ? RadixKeyKernel<KEY_SINGLE> : RadixKeyKernel<KEY_PACKED>;
    const cudaError_t err = EnsureDynamicSmem(reinterpret_cast<const void *>(kernel), kKeySmem);
    if (err != cudaSuccess) {
        return err;
    }
    const int grid = p.nTiles < DeviceSMCount() * 2 ? p.nTiles : DeviceSMCount() * 2;
    kernel<<<grid, kKeyThreads, kKeySmem, stream>>>(p, hist, regs);
    return cudaGetLastError();
}

cudaError_t LaunchRadixScatter(const AggLaunch &p, const RecLayout &l, int32_t bits, unsigned int *cursor,
    uint64_t *records, cudaStream_t stream)
{
    if (p.nTiles <= 0) {
        return cudaSuccess;
    }
    const size_t smem = (kScatterRows + (size_t(1) << bits)) * sizeof(unsigned int);
    auto kernel = p.key.kind == KEY_SINGLE ? RadixScatterKernel<KEY_SINGLE> : RadixScatterKernel<KEY_PACKED>;
    const cudaError_t err =
        EnsureDynamicSmem(reinterpret_cast<const void *>(kernel), (kScatterRows + kRadixFineParts) * sizeof(unsigned int));
    if (err != cudaSuccess) {
        return err;
    }
    const int steps = (p.nTiles + kScatterTiles - 1) / kScatterTiles;
    const int full = DeviceSMCount() * BlocksPerSM(reinterpret_cast<const void *>(kernel), kScatterThreads, smem);
    kernel<<<steps < full ? steps : full, kScatterThreads, smem, stream>>>(p, l, bits, cursor, records);
    return cudaGetLastError();
}

cudaError_t LaunchRadixAgg(const AggLaunch &p, const RecLayout &l, const RadixAgg &a, uint64_t *spill,
    unsigned int *nSpill, uint32_t spillCap, cudaStream_t stream)
{
    if (a.nUnits <= 0) {
        return cudaSuccess;
    }
    const SpillArgs sp{spill, nSpill, spillCap, nullptr, 0};
    auto kernel = p.key.kind == KEY_SINGLE ? RadixAggKernel<KEY_SINGLE> : RadixAggKernel<KEY_PACKED>;
    const cudaError_t err = EnsureDynamicSmem(reinterpret_cast<const void *>(kernel), kRadixSmemBytes);
    if (err != cudaSuccess) {
        return err;
    }
    const int grid = a.nUnits < DeviceSMCount() * 2 ? a.nUnits : DeviceSMCount() * 2;
    kernel<<<grid, kStepThreads, kRadixSmemBytes, stream>>>(p, l, a, sp);
    return cudaGetLastError();
}

cudaError_t LaunchRadixRetry(const AggLaunch &p, const RecLayout &l, const uint64_t *records, uint64_t *spill,
    unsigned int *nSpill, uint32_t spillCap, const uint64_t *spillIn, uint32_t nSpillIn, int gridBlocks,
    cudaStream_t stream)
{
    const SpillArgs sp{spill, nSpill, spillCap, spillIn, nSpillIn};
    auto kernel = p.key.kind == KEY_SINGLE ? RadixRetryKernel<KEY_SINGLE> : RadixRetryKernel<KEY_PACKED>;
    kernel<<<gridBlocks, 512, 0, stream>>>(p, l, records, sp);
    return cudaGetLastError();
}

}  // namespace omg
