// Hash aggregation kernels for sm_103a.
//
// Replaces the row loop of HashAggregationOperator::AddInput / Emplace
// (operator/aggregation/group_aggregation.cpp:320-406,811-890): find-or-insert the group of
// every row, then update its aggregate states (operations_hash_aggregator.h:16-76).
//
// Design:
//  * One persistent grid walks the tile list of many VectorBatches (host-pinned or HBM).
//  * Each CTA keeps a shared-memory pre-aggregation table; a row whose group is found or
//    placed there is updated with shared-memory atomics.  Rows that miss (table full) go to
//    the global open-addressing table with 64-bit atomicCAS insertion and global atomics.
//    At the end each CTA merges its shared table into the global one.
//  * States are exact or order-free: wrapping int64 sums, exact 128/192-bit sums kept as
//    separate positive and negative magnitudes (so Sum|x| is known for the sticky-overflow
//    rule), compensated double sums, and monotone min/max with a read-before-atomic filter.
//  * A row that cannot be placed within `maxProbe` probes is queued, never half-applied; the
//    host grows the table and re-runs the queue.  A shared-table entry that cannot be merged
//    is spilled as a partial record and merged after the growth.
#include <cstdint>
#include <cuda_runtime.h>

#include "agg_device.cuh"
#include "agg_extract.cuh"
#include "device_common.cuh"
#include "launch.h"
#include "plan.h"

namespace omg {
namespace {

constexpr int kAggThreads = 512;

// ------------------------------------------------------------------ partitioned tiles
// Partitioned launches process a tile in two passes.  Pass 1 resolves each of the thread's rows
// to a slot of the CTA's shared table (a row whose group does not fit, or a NULL / EMPTY key,
// goes through the generic global path at once).  Pass 2 walks the accumulators once per tile:
// the accumulator's kind and input width are dispatched once, then applied to the thread's rows,
// so the per-row work is the value load and the shared-memory atomic.
// Latency of those atomics bounds it (a third of the issue slots in use), so 64-bit words are added to in
// native 32-bit halves, a double sum's error costs two FP64 operations in place of six, and the four rows'
// loads go out together, once per input: 4M rows in 10,000 groups, six aggregates, 198 -> 166 us; 3M rows in
// 118 groups of a two-column key, 304 -> 205 us.  512 threads of eight rows each took 304 us for the former.
constexpr int kPartThreads = 1024;
constexpr int kPartRows = kTileRows / kPartThreads;
// Probes before a row goes to the global table.  With 8, one or two groups in a hundred never got a place at a
// load of 0.6, and all their rows met in a few global slots: 166 -> 118 us for 4M rows in 10,000 groups, and
// 4.0 -> 1.0 ms on a two-column key.
constexpr int kPartProbe = 32;

// A double into a sum in the shared table (AddDoubleState).
__device__ __forceinline__ void AddSharedDouble(uint64_t *w, double x, uint32_t arrival)
{
    if (arrival < kPlainSumRows) {
        atomicAdd(reinterpret_cast<double *>(w), x);
    } else {
        SharedAddCompensated(w, x);
    }
}

// The rows of a tile whose key hash wants(hash) takes; elsewhere(row) takes a row without a place in the table.
// kPlain: the first kPlainSumRows doubles of a slot are added plainly.
template <int kKind, bool kPlain, class Wants, class Elsewhere>
__device__ __forceinline__ void ProcessPartTile(const AggLaunch &p, const BatchDesc &b, const TileDesc &tile,
    uint64_t *sm, int smSlots, Wants wants, Elsewhere elsewhere)
{
    const int sw = p.smemStride;
    const int kw = p.table.keyWords;
    const BatchRows<kPartThreads> rows{b, static_cast<int64_t>(tile.row0) + threadIdx.x};
    int slot[kPartRows];          // index in the shared table
    uint32_t arrival[kPartRows];  // the row's COUNT_ALL arrival order in its slot (capped)
    uint32_t live = 0;            // bit k: row k has a slot
    {
        uint32_t use = 0;
#pragma unroll
        for (int k = 0; k < kPartRows; ++k) {
            use |= static_cast<int>(threadIdx.x) + k * kPartThreads < tile.rows ? 1u << k : 0u;
        }
        constexpr int kBatch = kKind == KEY_SINGLE ? kPartRows : 2;  // wide keys of four rows spill
#pragma unroll
        for (int k0 = 0; k0 < kPartRows; k0 += kBatch) {
            RowKey key[kBatch];
            ReadKeys<kKind, kBatch>(p.key, BatchRows<kPartThreads>{b, rows.row0 + k0 * kPartThreads}, use >> k0, key);
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                slot[k0 + k] = 0;
                arrival[k0 + k] = static_cast<uint32_t>(kPlainSumRows);
                if (!wants(key[k].hash)) {
                    use &= ~(1u << (k0 + k));
                }
                if (((use >> (k0 + k)) & 1u) != 0 && key[k].special < 0) {
                    slot[k0 + k] = SmemFind(sm, smSlots, sw, p.key, key[k], kKind, kPartProbe);
                    live |= slot[k0 + k] >= 0 ? 1u << (k0 + k) : 0u;
                }
            }
        }
        // Rows whose group is not in the shared table: the generic global path.
#pragma unroll 1
        for (uint32_t rest = use & ~live; rest != 0; rest &= rest - 1) {
            elsewhere(rows.row0 + (__ffs(rest) - 1) * kPartThreads);
        }
    }
    uint64_t *st = sm + kw;  // state words of slot i start at st + i * sw
    int input = -1;          // the input that has and, if loaded, bits are of
    bool loaded = false;
    uint64_t bits[kPartRows];
    uint32_t has = 0;        // the rows whose value is not NULL
    for (int a = 0; a < p.nAccs; ++a) {
        const AccSpec s = p.accs[a];
        if (s.kind == ACC_COUNT_ALL) {
#pragma unroll
            for (int k = 0; k < kPartRows; ++k) {
                if ((live >> k) & 1u) {
                    // A shared table counts the rows of one launch (< 2^32): a 32-bit add on the
                    // word's low half (little-endian) is exact and faster than a 64-bit one.
                    const unsigned int n = atomicAdd(LowHalf(st + slot[k] * sw + s.word), 1u);
                    arrival[k] = kPlain ? min(n, static_cast<unsigned int>(kPlainSumRows)) : arrival[k];
                }
            }
            continue;
        }
        if (s.input != input) {
            input = s.input;
            loaded = false;
            has = live;
            if (rows.Nullable(input)) {
                has &= ~rows.template Nulls<kPartRows>(input, live);
            }
        }
        const int width = s.kind == ACC_SMIN || s.kind == ACC_SMAX ? 4 : s.inWidth;
        if (!loaded && s.kind != ACC_NULLS && width <= 8) {
            loaded = true;
            LoadBitsRows<kPartRows>([&](int j) { return rows.At(input, width, j); }, width, has, bits);
        }
        uint64_t *base = st + s.word;
        switch (s.kind) {
            case ACC_NULLS:
#pragma unroll
                for (int k = 0; k < kPartRows; ++k) {
                    if (((live & ~has) >> k) & 1u) {
                        atomicAdd(LowHalf(base + slot[k] * sw), 1u);
                    }
                }
                break;
            case ACC_ISUM:
#pragma unroll
                for (int k = 0; k < kPartRows; ++k) {
                    if ((has >> k) & 1u) {
                        SharedAdd(base + slot[k] * sw, static_cast<uint64_t>(SignExtend(bits[k], s.inWidth)));
                    }
                }
                break;
            case ACC_WSUM2:
#pragma unroll
                for (int k = 0; k < kPartRows; ++k) {
                    if ((has >> k) & 1u) {
                        const int64_t x = SignExtend(bits[k], s.inWidth);
                        const uint64_t m = x >= 0 ? static_cast<uint64_t>(x) : 0ull - static_cast<uint64_t>(x);
                        uint64_t *side = base + slot[k] * sw + (x >= 0 ? 0 : 2);
                        SharedAdd(side, m & 0xffffffffull);
                        SharedAdd(side + 1, m >> 32);
                    }
                }
                break;
            case ACC_IMIN:
            case ACC_IMAX:
            case ACC_DMIN:
            case ACC_DMAX: {
                const bool isMin = s.kind == ACC_IMIN || s.kind == ACC_DMIN;
                const bool isInt = s.kind == ACC_IMIN || s.kind == ACC_IMAX;
#pragma unroll
                for (int k = 0; k < kPartRows; ++k) {
                    if (((has >> k) & 1u) == 0) {
                        continue;
                    }
                    int64_t x = SignExtend(bits[k], s.inWidth);
                    if (!isInt) {
                        const double d = AsDouble(bits[k], s.inKind, s.inWidth);
                        if (isnan(d)) {
                            continue;
                        }
                        x = OrderedFromDouble(d);
                    }
                    uint64_t *w = base + slot[k] * sw;
                    if (isMin) {
                        AtomicMinI64(w, x);
                    } else {
                        AtomicMaxI64(w, x);
                    }
                }
                break;
            }
            case ACC_DSUM:
#pragma unroll
                for (int k = 0; k < kPartRows; ++k) {
                    if ((has >> k) & 1u) {
                        AddSharedDouble(base + slot[k] * sw, AsDouble(bits[k], s.inKind, s.inWidth), arrival[k]);
                    }
                }
                break;
            default:  // decimal128 and string states
#pragma unroll 1
                for (uint32_t rest = has; rest != 0; rest &= rest - 1) {
                    const int k = __ffs(rest) - 1;
                    int at = slot[0];
                    uint64_t v = bits[0];
#pragma unroll
                    for (int j = 1; j < kPartRows; ++j) {
                        at = j == k ? slot[j] : at;
                        v = j == k ? bits[j] : v;
                    }
                    uint64_t *w = base + at * sw;
                    if (s.kind == ACC_SMIN || s.kind == ACC_SMAX) {
                        AtomicStrMinMax(p, input, w, SignExtend(v, 4), s.kind == ACC_SMIN);
                    } else {
                        ApplyWide(s, rows.At(input, 16, k), w);
                    }
                }
                break;
        }
    }
}

__device__ __forceinline__ void InitSharedSlots(const AggLaunch &p, uint64_t *smem, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        InitSlot(p, smem + static_cast<int64_t>(i) * p.smemStride);
    }
}

template <int kKind, bool kPart>
__device__ __forceinline__ void AggBody(const AggLaunch &p, const SpillArgs &sp, uint64_t *smem,
    unsigned int &newGroups)
{
    const int sw = p.table.slotWords;
    const int ss = p.smemStride;
    const int kw = p.table.keyWords;
    const int smSlots = (p.retryIn == nullptr && sp.spillIn == nullptr) ? p.smemSlots : 0;
    if (threadIdx.x == 0) {
        newGroups = 0;
    }
    InitSharedSlots(p, smem, smSlots);
    __syncthreads();

    if (p.retryIn != nullptr || sp.spillIn != nullptr) {
        const int64_t gtid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
        const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
        for (int64_t i = gtid; i < p.nRetryIn; i += stride) {
            unsigned long long e = p.retryIn[i];
            const int32_t bi = static_cast<int32_t>(e >> 32);
            const int64_t row = static_cast<int64_t>(e & 0xffffffffull);
            const BatchDesc &b = p.batches[bi];
            ProcessRow<kKind>(p, bi, b, row, LoadRow<kKind>(p, b, row), smem, 0, &newGroups);
        }
        for (int64_t i = gtid; i < sp.nSpillIn; i += stride) {
            MergeRecord<kKind>(p, sp, sp.spillIn + i * sw, &newGroups);
        }
    } else {
        // Two rows per thread per step: both rows' loads are issued before either is processed.
        int tFirst = blockIdx.x;
        int tEnd = p.nTiles;
        int tStep = gridDim.x;
        if (p.nParts > 0) {  // gridDim.x is a multiple of nParts
            const int q = blockIdx.x % p.nParts;
            tFirst = p.partTileStart[q] + blockIdx.x / p.nParts;
            tEnd = p.partTileStart[q + 1];
            tStep = gridDim.x / p.nParts;
        }
        if (kPart && smSlots > 0) {
            for (int t = tFirst; t < tEnd; t += tStep) {
                const TileDesc tile = p.tiles[t];
                const BatchDesc &b = p.batches[tile.batch];
                ProcessPartTile<kKind, true>(p, b, tile, smem, smSlots, [](uint64_t) { return true; }, [&](int64_t row) {
                    ProcessRow<kKind>(p, tile.batch, b, row, LoadRow<kKind>(p, b, row), smem, 0, &newGroups);
                });
            }
            tEnd = tFirst;  // done
        }
        for (int t = tFirst; t < tEnd; t += tStep) {
            const TileDesc tile = p.tiles[t];
            const BatchDesc &b = p.batches[tile.batch];
            for (int r = threadIdx.x; r < tile.rows; r += 2 * blockDim.x) {
                const int64_t row0 = static_cast<int64_t>(tile.row0) + r;
                const bool second = r + static_cast<int>(blockDim.x) < tile.rows;
                const RowIn a = LoadRow<kKind>(p, b, row0);
                RowIn c;
                if (second) {
                    c = LoadRow<kKind>(p, b, row0 + blockDim.x);
                }
                ProcessRow<kKind>(p, tile.batch, b, row0, a, smem, smSlots, &newGroups);
                if (second) {
                    ProcessRow<kKind>(p, tile.batch, b, row0 + blockDim.x, c, smem, smSlots, &newGroups);
                }
            }
        }
    }
    __syncthreads();

    // Merge the shared table into the global table.
    for (int i = threadIdx.x; i < smSlots; i += blockDim.x) {
        const uint64_t *slot = smem + static_cast<int64_t>(i) * ss;
        if (SlotOccupied(p.key, slot[0])) {
            MergeRecord<kKind>(p, sp, slot, &newGroups);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && newGroups != 0) {
        atomicAdd(p.table.groupCount, static_cast<unsigned long long>(newGroups));
    }
}

template <int kKind>
__global__ void __launch_bounds__(kAggThreads, 2) AggKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ SpillArgs sp)
{
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ unsigned int newGroups;
    AggBody<kKind, false>(p, sp, smem, newGroups);
}

// Partitioned launches: one 1024-thread CTA per SM with a shared table of up to
// kPartSmemBytes (the partition's groups).
constexpr size_t kPartSmemBytes = 200 * 1024;

template <int kKind>
__global__ void __launch_bounds__(kPartThreads, 1) AggPartKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ SpillArgs sp)
{
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ unsigned int newGroups;
    AggBody<kKind, true>(p, sp, smem, newGroups);
}

// ------------------------------------------------------------------ table maintenance
__global__ void InitTableKernel(AggTable t, int keyKind, const __grid_constant__ AggLaunch p)
{
    const uint64_t n = t.capacity + 2;
    for (uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s < n;
         s += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        uint64_t *slot = t.slots + s * t.slotWords;
        slot[0] = (keyKind == KEY_SINGLE) ? kEmptyKey : 0ull;
        for (int j = 1; j < t.keyWords; ++j) {
            slot[j] = 0;
        }
        InitStates(p.accs, p.nAccs, p.stateWords, slot + t.keyWords);
    }
    if (blockIdx.x == 0 && threadIdx.x < 2) {
        t.specialUsed[threadIdx.x] = 0;
    }
}

// Move every group of `from` into the (initialised, larger) table `to`.
__global__ void RehashKernel(AggTable from, AggTable to, const __grid_constant__ AggLaunch p)
{
    const uint64_t n = from.capacity + 2;
    for (uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s < n;
         s += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t *src = from.slots + s * from.slotWords;
        uint64_t *dst = nullptr;
        if (s >= from.capacity) {
            const int sp = static_cast<int>(s - from.capacity);
            if (from.specialUsed[sp] == 0) {
                continue;
            }
            to.specialUsed[sp] = 1;
            dst = to.slots + (to.capacity + sp) * to.slotWords;
        } else {
            if (!SlotOccupied(p.key, src[0])) {
                continue;
            }
            RowKey k;
            k.special = -1;
            k.w[0] = k.w[1] = k.w[2] = 0;
            if (p.key.kind == KEY_SINGLE) {
                k.w[0] = src[0];
                k.hash = Mix64(k.w[0]);
            } else {
                uint64_t h = 0x9e3779b97f4a7c15ull;
                for (int i = 0; i < p.key.words; ++i) {
                    k.w[i] = src[1 + i];
                    h = Mix64(h ^ k.w[i]);
                }
                k.hash = h;
            }
            bool inserted = false;
            int64_t g = GlobalFind(to, p.key, k, static_cast<int>(to.capacity < (1ull << 30) ? to.capacity : (1ull << 30)),
                p.error, &inserted, p.waitBudget, p.key.kind);
            if (g < 0) {
                SetError(p.error, 4);
                continue;
            }
            dst = to.slots + g * to.slotWords;
        }
        for (int j = to.keyWords; j < to.slotWords; ++j) {
            dst[j] = src[j];
        }
    }
}

__global__ void CountGroupsKernel(AggTable t, int keyKind, unsigned long long *out)
{
    unsigned int local = 0;
    for (uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; s < t.capacity;
         s += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t w = t.slots[s * t.slotWords];
        local += (keyKind == KEY_SINGLE) ? (w != kEmptyKey) : (w != 0 && w != kTagLocked);
    }
    for (int o = 16; o > 0; o >>= 1) {
        local += __shfl_down_sync(0xffffffffu, local, o);
    }
    if ((threadIdx.x & 31) == 0 && local != 0) {
        atomicAdd(out, static_cast<unsigned long long>(local));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(out, static_cast<unsigned long long>(t.specialUsed[0] + t.specialUsed[1]));
    }
}

// One output column of AlignSchema over the tiles of the input batches (row order kept).
__global__ void AlignColumnKernel(const BatchDesc *batches, const TileDesc *tiles, int32_t nTiles,
    const int64_t *tileOutRow, const AlignCol c, void *out, uint8_t *outNulls)
{
    for (int t = blockIdx.x; t < nTiles; t += gridDim.x) {
        const TileDesc tile = tiles[t];
        const BatchDesc &b = batches[tile.batch];
        const int64_t out0 = tileOutRow[t];
        const void *col = c.input >= 0 ? b.cols[c.input] : nullptr;
        const uint8_t *nulls = c.input >= 0 ? b.nulls[c.input] : nullptr;
        for (int r = threadIdx.x; r < tile.rows; r += blockDim.x) {
            const int64_t row = static_cast<int64_t>(tile.row0) + r;
            const uint64_t pos = static_cast<uint64_t>(out0 + r);
            const bool isNull = NullRO(nulls, row);
            switch (c.op) {
                case ALIGN_COPY:
                    if (c.inWidth == 16) {
                        static_cast<longlong2 *>(out)[pos] = __ldg(static_cast<const longlong2 *>(col) + row);
                    } else {
                        StoreWidth(out, pos, c.outWidth, LoadBitsRO(col, row, c.inWidth));
                    }
                    break;
                case ALIGN_INT:
                    StoreWidth(out, pos, c.outWidth,
                        static_cast<uint64_t>(SignExtend(LoadBitsRO(col, row, c.inWidth), c.inWidth)));
                    break;
                case ALIGN_DOUBLE: {
                    const double v = LoadAsDoubleRO(col, row, c.inKind, c.inWidth);
                    if (c.outWidth == 4) {
                        static_cast<float *>(out)[pos] = static_cast<float>(v);
                    } else {
                        static_cast<double *>(out)[pos] = v;
                    }
                    break;
                }
                case ALIGN_ONE:
                    static_cast<int64_t *>(out)[pos] = 1;
                    break;
                case ALIGN_VALID:
                    static_cast<int64_t *>(out)[pos] = isNull ? 0 : 1;
                    break;
                default:  // ALIGN_AVG_SUM
                    static_cast<double *>(out)[pos] = isNull ? 0.0 : LoadAsDoubleRO(col, row, c.inKind, c.inWidth);
            }
            if (isNull && outNulls != nullptr) {
                SetOutNull(outNulls, pos);
            }
        }
    }
}

__global__ void ExtractKernel(const __grid_constant__ AggExtract e)
{
    __shared__ unsigned int warpCounts[32];
    __shared__ unsigned long long blockBase;
    const AggTable &t = e.table;
    const uint64_t nSlots = t.capacity + 2;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int nWarps = blockDim.x >> 5;
    for (uint64_t base = static_cast<uint64_t>(blockIdx.x) * blockDim.x; base < nSlots;
         base += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t s = base + threadIdx.x;
        bool occ = false;
        const uint64_t *slot = nullptr;
        if (s < nSlots) {
            slot = t.slots + s * t.slotWords;
            occ = (s >= t.capacity) ? (t.specialUsed[s - t.capacity] != 0) : SlotOccupied(e.key, slot[0]);
        }
        const unsigned int ballot = __ballot_sync(0xffffffffu, occ);
        if (lane == 0) {
            warpCounts[warp] = __popc(ballot);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned int total = 0;
            for (int w = 0; w < nWarps; ++w) {
                unsigned int c = warpCounts[w];
                warpCounts[w] = total;
                total += c;
            }
            blockBase = total ? atomicAdd(e.outCount, static_cast<unsigned long long>(total)) : 0ull;
        }
        __syncthreads();
        if (occ) {
            const uint64_t pos = blockBase + warpCounts[warp] + __popc(ballot & ((1u << lane) - 1u));
            WriteGroup(e, t, s, slot, pos);
        }
        __syncthreads();
    }
}


__device__ __forceinline__ int PartOf(uint64_t hash, int partBits)
{
    return static_cast<int>((hash >> kPartShift) & ((1u << partBits) - 1u));
}

// ------------------------------------------------------------------ batched tasks
// Many independent aggregations (tasks) in one launch: task i is batch i and owns table
// taskTables[i] inside one slab.  AggTaskUnitsKernel adds up the tasks with few groups in shared tables, by units
// of their tiles; AggTasksKernel walks the tiles of the others (tiles of a task are adjacent).  The sketch runs one
// CTA per task, the count and the extraction one per kTaskChunkSlots slots of the tables.

// Rows per thread per step: their loads and first probes are issued together.
constexpr int kTaskRows = 1;

template <int kKind, int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) AggTasksKernel(const __grid_constant__ AggLaunch p)
{
    const int sw = p.table.slotWords;
    const int kw = p.table.keyWords;
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        const TileDesc tile = p.tiles[t];
        // A task that already overflowed its table is re-run exactly by the host: skip its rows.
        if (p.taskShared[tile.batch] != 0 || *reinterpret_cast<volatile uint32_t *>(p.taskFailed + tile.batch) != 0u) {
            continue;
        }
        const BatchDesc &b = p.batches[tile.batch];
        const AggTable tab = p.taskTables[tile.batch];
        for (int r0 = threadIdx.x; r0 < tile.rows; r0 += kThreads * kTaskRows) {
            RowIn in[kTaskRows];
            int64_t g[kTaskRows];
#pragma unroll
            for (int k = 0; k < kTaskRows; ++k) {
                const int r = r0 + k * kThreads;
                if (r < tile.rows) {
                    in[k] = LoadRow<kKind>(p, b, static_cast<int64_t>(tile.row0) + r);
                }
            }
#pragma unroll
            for (int k = 0; k < kTaskRows; ++k) {
                g[k] = -2;
                if (r0 + k * kThreads < tile.rows) {
                    bool inserted = false;
                    g[k] = GlobalFind(tab, p.key, in[k].k, p.maxProbe, p.error, &inserted, p.waitBudget, kKind);
                }
            }
#pragma unroll
            for (int k = 0; k < kTaskRows; ++k) {
                if (g[k] == -1) {
                    p.taskFailed[tile.batch] = 1u;
                } else if (g[k] >= 0) {
                    UpdateStates(p, b, static_cast<int64_t>(tile.row0) + r0 + k * kThreads, in[k],
                        tab.slots + g[k] * sw + kw);
                }
            }
        }
    }
}

// The tasks with few groups: a random request to L2 per row, probe and state word bounded the kernel above
// (5.3 ms for 58M rows in 400 tasks, at the 38 G/s that such requests go at), so here a CTA adds up a run of a
// task's rows in a shared table and merges that: 1.0 ms, and 1.9 above for the tasks left.  More groups than a
// table holds take up to eight runs over the keys, each for the rows of one partition; 16 runs took this
// kernel from 0.91 to 1.36 ms and the other from 2.15 to 1.58, 32 runs 2.14 and 1.29.  Doubles are compensated from
// the first one on: a group may have a slot in every unit of its task, and 64 plain rows in each.
template <int kKind>
__global__ void __launch_bounds__(kPartThreads, 1) AggTaskUnitsKernel(const __grid_constant__ AggLaunch p,
    const TaskUnit *units, int32_t nUnits, unsigned int *next)
{
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ unsigned int unitIndex;
    const int sw = p.table.slotWords;
    const int ss = p.smemStride;
    const int kw = p.table.keyWords;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            unitIndex = atomicAdd(next, 1u);
        }
        __syncthreads();
        if (unitIndex >= static_cast<unsigned int>(nUnits)) {
            break;
        }
        const TaskUnit unit = units[unitIndex];
        InitSharedSlots(p, smem, unit.slots);
        __syncthreads();
        const BatchDesc &b = p.batches[unit.task];
        const AggTable tab = p.taskTables[unit.task];
        // The state words of key k in the task's table, or null: the task has outgrown it.
        auto place = [&](const RowKey &k) {
            bool inserted = false;
            const int64_t g = GlobalFind(tab, p.key, k, p.maxProbe, p.error, &inserted, p.waitBudget, kKind);
            if (g == -1) {
                p.taskFailed[unit.task] = 1u;
            }
            return g >= 0 ? tab.slots + g * sw + kw : nullptr;
        };
        const volatile uint32_t *failed = p.taskFailed + unit.task;
        for (int t = unit.firstTile; t < unit.firstTile + unit.nTiles; ++t) {
            if (*failed != 0u) {
                break;  // the host re-runs the task exactly
            }
            ProcessPartTile<kKind, false>(p, b, p.tiles[t], smem, unit.slots,
                [&](uint64_t hash) { return PartOf(hash, unit.partBits) == unit.part; },
                [&](int64_t row) {
                    const RowIn in = LoadRow<kKind>(p, b, row);
                    uint64_t *st = place(in.k);
                    if (st != nullptr) {
                        UpdateStates(p, b, row, in, st);
                    }
                });
        }
        __syncthreads();
        for (int i = threadIdx.x; i < unit.slots && *failed == 0u; i += kPartThreads) {
            const uint64_t *slot = smem + static_cast<int64_t>(i) * ss;
            if (SlotOccupied(p.key, slot[0])) {
                uint64_t *st = place(RecordKey<kKind>(p, slot));
                if (st != nullptr) {
                    MergeStates(p, p.accs, p.nAccs, slot + kw, st);
                }
            }
        }
    }
}

// Per task: a sketch of up to kTaskSketchRows rows (stratified over the task's rows) in a
// shared-memory table; stats laid out as the operator's sketch (kSketchStats per task).
template <int kKind>
__global__ void __launch_bounds__(256) TaskSketchKernel(const __grid_constant__ AggLaunch p, int32_t nTasks,
    unsigned long long *stats)
{
    __shared__ unsigned long long keys[kTaskSketchSlots];
    __shared__ unsigned int counts[kTaskSketchSlots];
    __shared__ unsigned long long acc[kSketchStats];
    for (int task = blockIdx.x; task < nTasks; task += gridDim.x) {
        for (int i = threadIdx.x; i < kTaskSketchSlots; i += blockDim.x) {
            keys[i] = kEmptyKey;
            counts[i] = 0;
        }
        for (int i = threadIdx.x; i < kSketchStats; i += blockDim.x) {
            acc[i] = 0;
        }
        __syncthreads();
        const BatchDesc &b = p.batches[task];
        const int64_t rows = b.rows;
        const int n = static_cast<int>(rows < kTaskSketchRows ? rows : kTaskSketchRows);
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int64_t row = (static_cast<int64_t>(i) * rows) / n;
            const RowKey k = ReadKey(p.key, b, row, kKind);
            atomicAdd(&acc[0], 1ull);
            if (k.special >= 0) {
                atomicAdd(&acc[1], 1ull);
                continue;
            }
            const unsigned long long h = k.hash == kEmptyKey ? (k.hash ^ 1ull) : k.hash;
            uint32_t j = static_cast<uint32_t>(h) & (kTaskSketchSlots - 1);
            for (int probe = 0; probe < kTaskSketchSlots; ++probe) {
                const unsigned long long prev = atomicCAS(&keys[j], kEmptyKey, h);
                if (prev == kEmptyKey || prev == h) {
                    atomicAdd(&counts[j], 1u);
                    break;
                }
                j = (j + 1) & (kTaskSketchSlots - 1);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < kTaskSketchSlots; i += blockDim.x) {
            if (keys[i] == kEmptyKey) {
                continue;
            }
            const unsigned int c = counts[i];
            atomicAdd(&acc[2], 1ull);
            if (c == 1) {
                atomicAdd(&acc[3], 1ull);
            } else if (c == 2) {
                atomicAdd(&acc[4], 1ull);
            } else if (c == 3) {
                atomicAdd(&acc[5], 1ull);
            } else if (c < 8) {
                atomicAdd(&acc[6], 1ull);
            } else {
                atomicAdd(&acc[7], 1ull);
                atomicAdd(&acc[9], static_cast<unsigned long long>(c));
            }
            atomicMax(&acc[8], static_cast<unsigned long long>(c));
        }
        __syncthreads();
        for (int i = threadIdx.x; i < kSketchStats; i += blockDim.x) {
            stats[static_cast<int64_t>(task) * kSketchStats + i] = acc[i];
        }
        __syncthreads();
    }
}

// Tables are counted and extracted in chunks of kTaskChunkSlots slots, one CTA per chunk, because
// tasks differ a thousandfold in size: with one CTA per task the largest table's CTA ran on alone
// (400 tasks, 58 M rows, tables of up to 2^21 slots: count 2.35 ms and extraction 8.5 ms, and 4.7 and
// 16.5 ms more for two grown tasks; a run takes 5.9 ms with chunks, 33.8 ms without).
// Per task: occupied slots (special slots included), added up in counts (zeroed by the caller).
__global__ void __launch_bounds__(256) TaskCountKernel(const AggTable *tables, const TaskChunk *chunks,
    int32_t nChunks, int32_t keyKind, uint32_t *counts)
{
    KeySpec ks;
    ks.kind = keyKind;
    for (int c = blockIdx.x; c < nChunks; c += gridDim.x) {
        const TaskChunk ck = chunks[c];
        const AggTable t = tables[ck.task];
        const uint64_t first = static_cast<uint64_t>(ck.chunk) * kTaskChunkSlots;
        const uint64_t end = min(first + kTaskChunkSlots, t.capacity + 2);
        unsigned int mine = 0;
        for (uint64_t s = first + threadIdx.x; s < end; s += blockDim.x) {
            mine += (s >= t.capacity) ? (t.specialUsed[s - t.capacity] != 0)
                                      : SlotOccupied(ks, t.slots[s * t.slotWords]);
        }
        mine = __reduce_add_sync(0xffffffffu, mine);
        if ((threadIdx.x & 31) == 0 && mine != 0) {
            atomicAdd(&counts[ck.task], mine);
        }
    }
}

// Output region of each task: its group count rounded up to 64 rows, so that every region of the
// shared output columns starts on a byte of their null bitmaps.
__global__ void TaskPadKernel(const uint32_t *groups, int32_t nTasks, uint32_t *padded)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nTasks) {
        padded[t] = (groups[t] + 63u) / 64u * 64u;
    }
}

// The groups of each chunk, written to the task's region of the output columns: a warp reserves
// its rows at cursor[task] (which starts at the region's first row).
__global__ void __launch_bounds__(256) TaskExtractKernel(const __grid_constant__ AggExtract e, const AggTable *tables,
    const TaskChunk *chunks, int32_t nChunks, unsigned long long *cursor)
{
    const int lane = threadIdx.x & 31;
    for (int c = blockIdx.x; c < nChunks; c += gridDim.x) {
        const TaskChunk ck = chunks[c];
        const AggTable t = tables[ck.task];
        const uint64_t first = static_cast<uint64_t>(ck.chunk) * kTaskChunkSlots;
        const uint64_t end = min(first + kTaskChunkSlots, t.capacity + 2);
        for (uint64_t base = first + (threadIdx.x & ~31u); base < end; base += blockDim.x) {
            const uint64_t s = base + lane;
            bool occ = false;
            const uint64_t *slot = nullptr;
            if (s < end) {
                slot = t.slots + s * t.slotWords;
                occ = (s >= t.capacity) ? (t.specialUsed[s - t.capacity] != 0) : SlotOccupied(e.key, slot[0]);
            }
            const unsigned int ballot = __ballot_sync(0xffffffffu, occ);
            unsigned long long pos = 0;
            if (lane == 0 && ballot != 0) {
                pos = atomicAdd(&cursor[ck.task], static_cast<unsigned long long>(__popc(ballot)));
            }
            pos = __shfl_sync(0xffffffffu, pos, 0);
            if (occ) {
                WriteGroup(e, t, s, slot, pos + __popc(ballot & ((1u << lane) - 1u)));
            }
        }
    }
}

// ------------------------------------------------------------------ ordered overflow replay
// For a group whose sticky-overflow outcome depends on row order (|exact sum| within the
// bound but Sum|x| beyond it), the reference marks the sum overflowed as soon as one
// row-ordered prefix leaves the bound (sum_aggregator.h:43-49, sum_spark_decimal_aggregator.h:
// 16-66).  This kernel replays those groups' rows in arrival order (batch, then row) on one
// thread and records, per group and exact-SUM column, whether a prefix left the bound.
// It only runs when such groups exist.
__device__ __forceinline__ int64_t FindSlot(const AggTable &t, const KeySpec &ks, const RowKey &k)
{
    if (k.special >= 0) {
        return static_cast<int64_t>(t.capacity) + k.special;
    }
    const uint64_t mask = t.capacity - 1;
    uint64_t i = k.hash & mask;
    const uint64_t tag = PublishedTag(k.hash);
    for (uint64_t probe = 0; probe < t.capacity; ++probe) {
        const uint64_t *slot = t.slots + i * t.slotWords;
        if (ks.kind == KEY_SINGLE) {
            if (slot[0] == k.w[0]) {
                return static_cast<int64_t>(i);
            }
            if (slot[0] == kEmptyKey) {
                return -1;
            }
        } else {
            if (slot[0] == 0) {
                return -1;
            }
            if (slot[0] == tag) {
                bool eq = true;
                for (int j = 0; j < ks.words; ++j) {
                    eq = eq && (slot[1 + j] == k.w[j]);
                }
                if (eq) {
                    return static_cast<int64_t>(i);
                }
            }
        }
        i = (i + 1) & mask;
    }
    return -1;
}

__global__ void OrderedOverflowKernel(const __grid_constant__ AggLaunch p, int32_t nBatches,
    const __grid_constant__ AggExtract e, const unsigned long long *ambSlots, uint32_t nAmb, int32_t *denseOf,
    uint64_t *prefix, uint8_t *forced)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) {
        return;
    }
    for (uint32_t i = 0; i < nAmb; ++i) {
        denseOf[ambSlots[i]] = static_cast<int32_t>(i);
    }
    for (int32_t bi = 0; bi < nBatches; ++bi) {
        const BatchDesc &b = p.batches[bi];
        for (int64_t row = 0; row < b.rows; ++row) {
            const RowKey k = ReadKey(p.key, b, row, p.key.kind);
            const int64_t slot = FindSlot(p.table, p.key, k);
            if (slot < 0 || denseOf[slot] < 0) {
                continue;
            }
            const int32_t d = denseOf[slot];
            for (int o = 0; o < e.nOut; ++o) {
                const OutSpec &os = e.out[o];
                if (os.kind != OUT_SUM_EXACT && os.kind != OUT_AVG_DEC) {
                    continue;
                }
                const uint8_t bit = static_cast<uint8_t>(1u << os.pad);
                if (forced[slot] & bit) {
                    continue;  // sticky: no further additions once overflowed
                }
                const AccSpec &acc = e.accs[os.src];
                if (RowIsNull(b.nulls[acc.input], row)) {
                    continue;
                }
                uint64_t x0, x1, x2;
                if (acc.kind == ACC_WSUM3) {
                    const uint64_t *v = static_cast<const uint64_t *>(b.cols[acc.input]) + 2 * row;
                    x0 = v[0];
                    x1 = v[1];
                    x2 = (static_cast<int64_t>(x1) < 0) ? ~0ull : 0ull;
                } else {
                    const int64_t v = LoadInt(b.cols[acc.input], row, acc.inWidth);
                    x0 = static_cast<uint64_t>(v);
                    x1 = x2 = (v < 0) ? ~0ull : 0ull;
                }
                uint64_t *pw = prefix + (static_cast<int64_t>(d) * 8 + os.pad) * 3;
                uint64_t a[3] = {pw[0], pw[1], pw[2]};
                uint64_t x[3] = {x0, x1, x2};
                uint64_t r[3];
                Add192(a, x, r);
                pw[0] = r[0];
                pw[1] = r[1];
                pw[2] = r[2];
                const bool neg = static_cast<int64_t>(r[2]) < 0;
                uint64_t mag[3];
                if (neg) {
                    const uint64_t zero[3] = {0, 0, 0};
                    Sub192(zero, r, mag);
                } else {
                    mag[0] = r[0];
                    mag[1] = r[1];
                    mag[2] = r[2];
                }
                if (ExceedsBound(mag, neg, os.boundKind)) {
                    forced[slot] |= bit;
                }
            }
        }
    }
}

// ------------------------------------------------------------------ hash partitioning
// Warp-aggregated increment of counter[part]: lanes with the same part elect one leader that adds
// the group's size; returns this lane's rank within its group plus the counter's old value.
__device__ __forceinline__ unsigned int WarpAggAdd(unsigned int *counter, int part, unsigned int active)
{
    const unsigned int peers = __match_any_sync(active, part);
    const int leader = __ffs(peers) - 1;
    const int lane = threadIdx.x & 31;
    unsigned int base = 0;
    if (lane == leader) {
        base = atomicAdd(&counter[part], static_cast<unsigned int>(__popc(peers)));
    }
    base = __shfl_sync(peers, base, leader);
    return base + __popc(peers & ((1u << lane) - 1u));
}

constexpr int kHistThreads = 512;
constexpr int kHistRows = 4;  // rows per thread per step: their key loads are in flight together (31 -> 24 us, 4M)

template <int kKind>
__global__ void __launch_bounds__(kHistThreads) PartHistKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ PartArgs a)
{
    __shared__ unsigned int h[kMaxParts];
    const int nParts = 1 << a.partBits;
    for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
        h[i] = 0;
    }
    __syncthreads();
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        const TileDesc tile = p.tiles[t];
        const BatchDesc &b = p.batches[tile.batch];
        for (int r0 = 0; r0 < tile.rows; r0 += kHistRows * kHistThreads) {
            uint32_t use = 0;
#pragma unroll
            for (int j = 0; j < kHistRows; ++j) {
                use |= r0 + j * kHistThreads + static_cast<int>(threadIdx.x) < tile.rows ? 1u << j : 0u;
            }
            RowKey key[kHistRows];
            ReadKeys<kKind, kHistRows>(p.key,
                BatchRows<kHistThreads>{b, static_cast<int64_t>(tile.row0) + r0 + threadIdx.x}, use, key);
#pragma unroll
            for (int j = 0; j < kHistRows; ++j) {
                const bool live = ((use >> j) & 1u) != 0;
                const unsigned int active = __ballot_sync(0xffffffffu, live);
                if (live) {
                    WarpAggAdd(h, PartOf(key[j].hash, a.partBits), active);
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
        if (h[i] != 0) {
            atomicAdd(&a.hist[i], static_cast<unsigned long long>(h[i]));
        }
    }
}

// One block: partition offsets (64-row aligned so every partition's NULL bitmap starts on a
// byte), the cursors, one batch descriptor per partition and the partitions' tiles.
__global__ void PartLayoutKernel(const __grid_constant__ PartArgs a)
{
    __shared__ unsigned long long offset[kMaxParts];
    const int nParts = 1 << a.partBits;
    if (threadIdx.x == 0) {
        unsigned long long off = 0;
        int tiles = 0;
        for (int q = 0; q < nParts; ++q) {
            offset[q] = off;
            a.cursor[q] = off;
            off += (a.hist[q] + 63) / 64 * 64;
            a.partTileStart[q] = tiles;
            tiles += static_cast<int>((a.hist[q] + kTileRows - 1) / kTileRows);
        }
        a.partTileStart[nParts] = tiles;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nParts; q += blockDim.x) {
        BatchDesc d;
        for (int i = 0; i < kMaxInputs; ++i) {
            d.cols[i] = nullptr;
            d.nulls[i] = nullptr;
            d.offs[i] = nullptr;
        }
        for (int i = 0; i < a.nInputs; ++i) {
            d.cols[i] = static_cast<char *>(a.cols[i]) + offset[q] * a.width[i];
            d.nulls[i] = a.nulls[i] != nullptr ? reinterpret_cast<const uint8_t *>(a.nulls[i]) + offset[q] / 8 : nullptr;
        }
        d.rows = static_cast<int64_t>(a.hist[q]);
        d.rowBase = static_cast<int64_t>(offset[q]);
        a.partBatches[q] = d;
        const int first = a.partTileStart[q];
        const int n = a.partTileStart[q + 1] - first;
        for (int k = 0; k < n && first + k < a.maxTiles; ++k) {
            TileDesc td;
            td.batch = q;
            td.row0 = k * kTileRows;
            td.rows = static_cast<int32_t>(min(static_cast<unsigned long long>(kTileRows), a.hist[q] - k * kTileRows));
            td.pad = 0;
            a.partTiles[first + k] = td;
        }
    }
}

__device__ __forceinline__ void CopyInput(const void *src, int64_t row, void *dst, uint64_t pos, int width)
{
    switch (width) {
        case 1:
            static_cast<uint8_t *>(dst)[pos] = static_cast<uint8_t>(__ldg(static_cast<const unsigned char *>(src) + row));
            break;
        case 2:
            static_cast<uint16_t *>(dst)[pos] = static_cast<uint16_t>(__ldg(static_cast<const unsigned short *>(src) + row));
            break;
        case 4:
            static_cast<uint32_t *>(dst)[pos] = __ldg(static_cast<const unsigned int *>(src) + row);
            break;
        case 8:
            static_cast<uint64_t *>(dst)[pos] = __ldg(static_cast<const unsigned long long *>(src) + row);
            break;
        default: {
            const ulonglong2 v = __ldg(static_cast<const ulonglong2 *>(src) + row);
            static_cast<ulonglong2 *>(dst)[pos] = v;
            break;
        }
    }
}

// Input `input` of N rows (bit j of `use`) to places pos[j]; all loads come before the stores.
template <int N, class Rows>
__device__ __forceinline__ void CopyRows(const Rows &rows, int input, int width, uint32_t use, void *dst,
    const uint64_t (&pos)[N])
{
    uint64_t v[N];
    if (width == 16) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            LoadBitsRows<N>([&](int j) { return rows.At(input, 16, j) + 8 * half; }, 8, use, v);
#pragma unroll
            for (int j = 0; j < N; ++j) {
                if ((use >> j) & 1u) {
                    static_cast<uint64_t *>(dst)[2 * pos[j] + half] = v[j];
                }
            }
        }
        return;
    }
    LoadBitsRows<N>([&](int j) { return rows.At(input, width, j); }, width, use, v);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        if (((use >> j) & 1u) == 0) {
            continue;
        }
        switch (width) {
            case 1:
                static_cast<uint8_t *>(dst)[pos[j]] = static_cast<uint8_t>(v[j]);
                break;
            case 2:
                static_cast<uint16_t *>(dst)[pos[j]] = static_cast<uint16_t>(v[j]);
                break;
            case 4:
                static_cast<uint32_t *>(dst)[pos[j]] = static_cast<uint32_t>(v[j]);
                break;
            default:
                static_cast<uint64_t *>(dst)[pos[j]] = v[j];
                break;
        }
    }
}

// Per tile: partition of every row, one cursor reservation per partition, then each row's
// inputs copied to its partition (rows of a partition from one warp land contiguously).
constexpr int kScatterThreads = 512;
constexpr int kScatterRows = kTileRows / kScatterThreads;

template <int kKind>
__global__ void __launch_bounds__(kScatterThreads) PartScatterKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ PartArgs a)
{
    __shared__ unsigned int cnt[kMaxParts];
    __shared__ unsigned long long base[kMaxParts];
    const int nParts = 1 << a.partBits;
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        const TileDesc tile = p.tiles[t];
        const BatchDesc &b = p.batches[tile.batch];
        for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
            cnt[i] = 0;
        }
        __syncthreads();
        const BatchRows<kScatterThreads> rows{b, static_cast<int64_t>(tile.row0) + threadIdx.x};
        uint32_t use = 0;
#pragma unroll
        for (int j = 0; j < kScatterRows; ++j) {
            use |= static_cast<int>(threadIdx.x) + j * kScatterThreads < tile.rows ? 1u << j : 0u;
        }
        uint32_t place[kScatterRows];  // partition << 16 | rank among the tile's rows of the partition
        {
            RowKey key[kScatterRows];
            ReadKeys<kKind, kScatterRows>(p.key, rows, use, key);
#pragma unroll
            for (int j = 0; j < kScatterRows; ++j) {
                const bool live = ((use >> j) & 1u) != 0;
                const unsigned int active = __ballot_sync(0xffffffffu, live);
                place[j] = 0;
                if (live) {
                    const int q = PartOf(key[j].hash, a.partBits);
                    place[j] = (static_cast<uint32_t>(q) << 16) | WarpAggAdd(cnt, q, active);
                }
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
            base[i] = cnt[i] != 0 ? atomicAdd(&a.cursor[i], static_cast<unsigned long long>(cnt[i])) : 0ull;
        }
        __syncthreads();
        uint64_t pos[kScatterRows];
#pragma unroll
        for (int j = 0; j < kScatterRows; ++j) {
            pos[j] = base[place[j] >> 16] + (place[j] & 0xffffu);
        }
        for (int i = 0; i < a.nInputs; ++i) {
            CopyRows<kScatterRows>(rows, i, a.width[i], use, a.cols[i], pos);
            if (a.nulls[i] != nullptr && rows.Nullable(i)) {
                const uint32_t null = rows.template Nulls<kScatterRows>(i, use);
#pragma unroll
                for (int j = 0; j < kScatterRows; ++j) {
                    if ((null >> j) & 1u) {
                        atomicOr(&a.nulls[i][pos[j] >> 5], 1u << (pos[j] & 31));
                    }
                }
            }
        }
        __syncthreads();
    }
}

// ---- stable partitioning (order-dependent plans) ----
// Per tile: rows per partition.
template <int kKind>
__global__ void __launch_bounds__(512) PartTileHistKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ PartArgs a)
{
    __shared__ unsigned int h[kMaxParts];
    const int nParts = 1 << a.partBits;
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
            h[i] = 0;
        }
        __syncthreads();
        const TileDesc tile = p.tiles[t];
        const BatchDesc &b = p.batches[tile.batch];
        for (int r = threadIdx.x; r < tile.rows; r += blockDim.x) {
            atomicAdd(&h[PartOf(ReadKey(p.key, b, static_cast<int64_t>(tile.row0) + r, kKind).hash, a.partBits)], 1u);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
            a.tileHist[static_cast<int64_t>(t) * nParts + i] = h[i];
        }
        __syncthreads();
    }
}

// One block per partition: the exclusive prefix of its per-tile counts in tile order (in place)
// and its total rows.
__global__ void __launch_bounds__(1024) PartTileScanKernel(const __grid_constant__ PartArgs a, int32_t nTiles)
{
    __shared__ unsigned long long warpSum[32];
    __shared__ unsigned long long carry;
    const int q = blockIdx.x;
    const int nParts = 1 << a.partBits;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        carry = 0;
    }
    __syncthreads();
    for (int t0 = 0; t0 < nTiles; t0 += blockDim.x) {
        const int t = t0 + static_cast<int>(threadIdx.x);
        const unsigned long long v = t < nTiles ? a.tileHist[static_cast<int64_t>(t) * nParts + q] : 0ull;
        unsigned long long incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, d);
            incl += lane >= d ? u : 0ull;
        }
        if (lane == 31) {
            warpSum[warp] = incl;
        }
        __syncthreads();
        if (warp == 0) {
            const unsigned long long w = lane < static_cast<int>(blockDim.x >> 5) ? warpSum[lane] : 0ull;
            unsigned long long wi = w;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long u = __shfl_up_sync(0xffffffffu, wi, d);
                wi += lane >= d ? u : 0ull;
            }
            warpSum[lane] = wi - w;  // exclusive prefix of the warps
        }
        __syncthreads();
        const unsigned long long excl = carry + warpSum[warp] + incl - v;
        if (t < nTiles) {
            a.tileHist[static_cast<int64_t>(t) * nParts + q] = static_cast<unsigned int>(excl);
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) {
            carry = excl + v;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        a.hist[q] = carry;
    }
}

// Per tile: each row to its partition at the tile's offset there plus its rank among the tile's
// earlier rows of that partition (rounds in order; within a round, warps in order, then lanes).
template <int kKind>
__global__ void __launch_bounds__(kScatterThreads) PartScatterStableKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ PartArgs a)
{
    constexpr int kWarps = kScatterThreads / 32;
    __shared__ unsigned int warpCnt[kWarps][kMaxParts];  // counts, then exclusive prefixes over warps
    __shared__ unsigned int roundTotal[kMaxParts];
    __shared__ unsigned long long running[kMaxParts];
    const int nParts = 1 << a.partBits;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned int below = (1u << lane) - 1u;
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        const TileDesc tile = p.tiles[t];
        const BatchDesc &b = p.batches[tile.batch];
        for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
            running[i] = a.cursor[i] + a.tileHist[static_cast<int64_t>(t) * nParts + i];
        }
        for (int j = 0; j < kScatterRows; ++j) {
            for (int i = threadIdx.x; i < kWarps * kMaxParts; i += blockDim.x) {
                warpCnt[i / kMaxParts][i % kMaxParts] = 0;
            }
            __syncthreads();
            const int r = j * kScatterThreads + static_cast<int>(threadIdx.x);
            const bool live = r < tile.rows;
            const unsigned int active = __ballot_sync(0xffffffffu, live);
            int q = 0;
            unsigned int peers = 0;
            if (live) {
                q = PartOf(ReadKey(p.key, b, static_cast<int64_t>(tile.row0) + r, kKind).hash, a.partBits);
                peers = __match_any_sync(active, q);
                if ((peers & below) == 0) {
                    warpCnt[warp][q] = __popc(peers);  // written by the partition's first lane
                }
            }
            __syncthreads();
            for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
                unsigned int acc = 0;
                for (int w = 0; w < kWarps; ++w) {
                    const unsigned int c = warpCnt[w][i];
                    warpCnt[w][i] = acc;
                    acc += c;
                }
                roundTotal[i] = acc;
            }
            __syncthreads();
            if (live) {
                const uint64_t pos = running[q] + warpCnt[warp][q] + __popc(peers & below);
                const int64_t row = static_cast<int64_t>(tile.row0) + r;
                for (int i = 0; i < a.nInputs; ++i) {
                    CopyInput(b.cols[i], row, a.cols[i], pos, a.width[i]);
                    if (a.nulls[i] != nullptr && RowIsNull(b.nulls[i], row)) {
                        atomicOr(&a.nulls[i][pos >> 5], 1u << (pos & 31));
                    }
                }
            }
            __syncthreads();
            for (int i = threadIdx.x; i < nParts; i += blockDim.x) {
                running[i] += roundTotal[i];
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ key sketch
// A sample of the rows, stratified over the tiles of the launch (sample s reads a hashed row of
// tile s * nTiles / nSample), is hashed into an open-addressing table of (hash, count);
// SketchStatsKernel then summarises the counts.
template <int kKind>
__global__ void SketchKernel(const __grid_constant__ AggLaunch p, int32_t nSample, unsigned long long *tabKeys,
    unsigned int *tabCounts, unsigned long long *stats)
{
    const uint32_t mask = kSketchCap - 1;
    unsigned long long seen = 0, special = 0;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nSample; s += gridDim.x * blockDim.x) {
        const int t = static_cast<int>((static_cast<int64_t>(s) * p.nTiles) / nSample);
        const TileDesc tile = p.tiles[t];
        if (tile.rows <= 0) {
            continue;
        }
        const int off = static_cast<int>(Mix64(static_cast<uint64_t>(s)) % static_cast<uint64_t>(tile.rows));
        const RowKey k = ReadKey(p.key, p.batches[tile.batch], static_cast<int64_t>(tile.row0) + off, kKind);
        ++seen;
        if (k.special >= 0) {
            ++special;
            continue;
        }
        const unsigned long long h = k.hash == kEmptyKey ? (k.hash ^ 1ull) : k.hash;
        uint32_t i = static_cast<uint32_t>(h) & mask;
        for (int probe = 0; probe < kSketchCap; ++probe) {
            const unsigned long long prev = atomicCAS(&tabKeys[i], kEmptyKey, h);
            if (prev == kEmptyKey || prev == h) {
                atomicAdd(&tabCounts[i], 1u);
                break;
            }
            i = (i + 1) & mask;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        seen += __shfl_down_sync(0xffffffffu, seen, o);
        special += __shfl_down_sync(0xffffffffu, special, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&stats[0], seen);
        if (special != 0) {
            atomicAdd(&stats[1], special);
        }
    }
}

__global__ void SketchInitKernel(unsigned long long *tabKeys, unsigned int *tabCounts, unsigned long long *stats)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kSketchCap; i += gridDim.x * blockDim.x) {
        tabKeys[i] = kEmptyKey;
        tabCounts[i] = 0;
        if (i < kSketchStats) {
            stats[i] = 0;
        }
    }
}

__global__ void SketchStatsKernel(const unsigned long long *tabKeys, const unsigned int *tabCounts,
    unsigned long long *stats)
{
    unsigned long long v[7] = {0, 0, 0, 0, 0, 0, 0};  // d, f1, f2, f3, f4-7, f8+, heavy rows
    unsigned long long mx = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kSketchCap; i += gridDim.x * blockDim.x) {
        if (tabKeys[i] == kEmptyKey) {
            continue;
        }
        const unsigned int c = tabCounts[i];
        v[0] += 1;
        v[1] += c == 1;
        v[2] += c == 2;
        v[3] += c == 3;
        v[4] += (c >= 4 && c < 8);
        v[5] += c >= 8;
        v[6] += c >= 8 ? c : 0;
        mx = c > mx ? c : mx;
    }
#pragma unroll
    for (int j = 0; j < 7; ++j) {
        for (int o = 16; o > 0; o >>= 1) {
            v[j] += __shfl_down_sync(0xffffffffu, v[j], o);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long om = __shfl_down_sync(0xffffffffu, mx, o);
        mx = om > mx ? om : mx;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&stats[2], v[0]);
        atomicAdd(&stats[3], v[1]);
        atomicAdd(&stats[4], v[2]);
        atomicAdd(&stats[5], v[3]);
        atomicAdd(&stats[6], v[4]);
        atomicAdd(&stats[7], v[5]);
        atomicMax(&stats[8], mx);
        atomicAdd(&stats[9], v[6]);
    }
}

int NumSMs() { return DeviceSMCount(); }

}  // namespace

cudaError_t LaunchAggInitTable(const AggLaunch &p, cudaStream_t stream)
{
    const uint64_t n = p.table.capacity + 2;
    const int threads = 256;
    uint64_t blocks = (n + threads - 1) / threads;
    const uint64_t maxBlocks = static_cast<uint64_t>(NumSMs()) * 16;
    if (blocks > maxBlocks) {
        blocks = maxBlocks;
    }
    InitTableKernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(p.table, p.key.kind, p);
    return cudaGetLastError();
}

cudaError_t LaunchAggRehash(const AggLaunch &p, const AggTable &from, const AggTable &to, cudaStream_t stream)
{
    const uint64_t n = from.capacity + 2;
    const int threads = 256;
    uint64_t blocks = (n + threads - 1) / threads;
    const uint64_t maxBlocks = static_cast<uint64_t>(NumSMs()) * 16;
    if (blocks > maxBlocks) {
        blocks = maxBlocks;
    }
    RehashKernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(from, to, p);
    return cudaGetLastError();
}

cudaError_t LaunchAgg(const AggLaunch &p, uint64_t *spill, unsigned int *nSpill, uint32_t spillCap,
    const uint64_t *spillIn, uint32_t nSpillIn, int gridBlocks, cudaStream_t stream)
{
    SpillArgs sp{spill, nSpill, spillCap, spillIn, nSpillIn};
    const size_t smemBytes = static_cast<size_t>(p.smemSlots) * p.smemStride * sizeof(uint64_t);
    if (p.nParts > 0) {
        if (smemBytes > kPartSmemBytes) {
            return cudaErrorInvalidValue;
        }
        auto pk = p.key.kind == KEY_SINGLE ? AggPartKernel<KEY_SINGLE> : AggPartKernel<KEY_PACKED>;
        cudaError_t err = EnsureDynamicSmem(reinterpret_cast<const void *>(pk), kPartSmemBytes);
        if (err != cudaSuccess) {
            return err;
        }
        const int perPart = NumSMs() / p.nParts > 0 ? NumSMs() / p.nParts : 1;
        pk<<<perPart * p.nParts, kPartThreads, smemBytes, stream>>>(p, sp);
        return cudaGetLastError();
    }
    auto kernel = p.key.kind == KEY_SINGLE ? AggKernel<KEY_SINGLE> : AggKernel<KEY_PACKED>;
    cudaError_t err = EnsureDynamicSmem(reinterpret_cast<const void *>(kernel), smemBytes);
    if (err != cudaSuccess) {
        return err;
    }
    if (gridBlocks <= 0) {
        gridBlocks = NumSMs() * BlocksPerSM(reinterpret_cast<const void *>(kernel), kAggThreads, smemBytes);
    }
    kernel<<<gridBlocks, kAggThreads, smemBytes, stream>>>(p, sp);
    return cudaGetLastError();
}

cudaError_t LaunchAggCount(const AggTable &t, int keyKind, unsigned long long *out, cudaStream_t stream)
{
    const int threads = 256;
    uint64_t blocks = (t.capacity + threads - 1) / threads;
    const uint64_t maxBlocks = static_cast<uint64_t>(NumSMs()) * 8;
    if (blocks > maxBlocks) {
        blocks = maxBlocks;
    }
    if (blocks == 0) {
        blocks = 1;
    }
    CountGroupsKernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(t, keyKind, out);
    return cudaGetLastError();
}

cudaError_t LaunchAggExtract(const AggExtract &e, cudaStream_t stream)
{
    const int threads = 256;
    const uint64_t n = e.table.capacity + 2;
    uint64_t blocks = (n + threads - 1) / threads;
    const uint64_t maxBlocks = static_cast<uint64_t>(NumSMs()) * 8;
    if (blocks > maxBlocks) {
        blocks = maxBlocks;
    }
    ExtractKernel<<<static_cast<unsigned>(blocks), threads, 0, stream>>>(e);
    return cudaGetLastError();
}

cudaError_t LaunchAggOrdered(const AggLaunch &p, int32_t nBatches, const AggExtract &e,
    const unsigned long long *ambSlots, uint32_t nAmb, uint8_t *forced, cudaStream_t stream)
{
    const uint64_t nSlots = p.table.capacity + 2;
    int32_t *denseOf = nullptr;
    uint64_t *prefix = nullptr;
    cudaError_t err = cudaMallocAsync(reinterpret_cast<void **>(&denseOf), nSlots * sizeof(int32_t), stream);
    if (err != cudaSuccess) {
        return err;
    }
    err = cudaMallocAsync(reinterpret_cast<void **>(&prefix), static_cast<size_t>(nAmb) * 8 * 3 * sizeof(uint64_t) + 8,
        stream);
    if (err != cudaSuccess) {
        cudaFreeAsync(denseOf, stream);
        return err;
    }
    cudaMemsetAsync(denseOf, 0xff, nSlots * sizeof(int32_t), stream);
    cudaMemsetAsync(prefix, 0, static_cast<size_t>(nAmb) * 8 * 3 * sizeof(uint64_t) + 8, stream);
    OrderedOverflowKernel<<<1, 1, 0, stream>>>(p, nBatches, e, ambSlots, nAmb, denseOf, prefix, forced);
    err = cudaGetLastError();
    cudaFreeAsync(denseOf, stream);
    cudaFreeAsync(prefix, stream);
    return err;
}

cudaError_t LaunchAggTaskSketch(const AggLaunch &p, int32_t nTasks, unsigned long long *stats, cudaStream_t stream)
{
    if (nTasks <= 0) {
        return cudaSuccess;
    }
    const int grid = nTasks < NumSMs() * 8 ? nTasks : NumSMs() * 8;
    if (p.key.kind == KEY_SINGLE) {
        TaskSketchKernel<KEY_SINGLE><<<grid, 256, 0, stream>>>(p, nTasks, stats);
    } else {
        TaskSketchKernel<KEY_PACKED><<<grid, 256, 0, stream>>>(p, nTasks, stats);
    }
    return cudaGetLastError();
}

namespace {
// Launch shapes the autotuner chooses from: threads per CTA and the CTAs per SM the kernel is
// compiled for (the persistent grid is that many CTAs on every SM).
using TasksKernelFn = void (*)(AggLaunch);
struct TasksVariant {
    int32_t threads;
    int32_t blocksPerSM;
    TasksKernelFn single;
    TasksKernelFn packed;
};
const TasksVariant kTasksVariants[] = {
    {128, 8, AggTasksKernel<KEY_SINGLE, 128, 8>, AggTasksKernel<KEY_PACKED, 128, 8>},
    {256, 4, AggTasksKernel<KEY_SINGLE, 256, 4>, AggTasksKernel<KEY_PACKED, 256, 4>},
    {512, 2, AggTasksKernel<KEY_SINGLE, 512, 2>, AggTasksKernel<KEY_PACKED, 512, 2>},
    {1024, 1, AggTasksKernel<KEY_SINGLE, 1024, 1>, AggTasksKernel<KEY_PACKED, 1024, 1>},
};
}  // namespace

int32_t AggTasksVariants() { return static_cast<int32_t>(sizeof(kTasksVariants) / sizeof(kTasksVariants[0])); }

void AggTasksVariantShape(int32_t v, int32_t *threads, int32_t *blocksPerSM)
{
    *threads = kTasksVariants[v].threads;
    *blocksPerSM = kTasksVariants[v].blocksPerSM;
}

cudaError_t LaunchAggTasks(const AggLaunch &p, int32_t variant, cudaStream_t stream)
{
    if (p.nTiles <= 0) {
        return cudaSuccess;
    }
    if (variant < 0 || variant >= AggTasksVariants()) {
        return cudaErrorInvalidValue;
    }
    const TasksVariant &v = kTasksVariants[variant];
    int perSM = BlocksPerSM(reinterpret_cast<const void *>(p.key.kind == KEY_SINGLE ? v.single : v.packed), v.threads, 0);
    perSM = perSM > v.blocksPerSM ? v.blocksPerSM : perSM;
    int grid = NumSMs() * perSM;
    if (grid > p.nTiles) {
        grid = p.nTiles;
    }
    (p.key.kind == KEY_SINGLE ? v.single : v.packed)<<<grid, v.threads, 0, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t LaunchAggTaskUnits(const AggLaunch &p, const TaskUnit *units, int32_t nUnits, unsigned int *next,
    cudaStream_t stream)
{
    if (nUnits <= 0) {
        return cudaSuccess;
    }
    auto kernel = p.key.kind == KEY_SINGLE ? AggTaskUnitsKernel<KEY_SINGLE> : AggTaskUnitsKernel<KEY_PACKED>;
    cudaError_t err = EnsureDynamicSmem(reinterpret_cast<const void *>(kernel), kPartSmemBytes);
    if (err == cudaSuccess) {
        err = cudaMemsetAsync(next, 0, sizeof(*next), stream);
    }
    if (err != cudaSuccess) {
        return err;
    }
    kernel<<<nUnits < NumSMs() ? nUnits : NumSMs(), kPartThreads, kPartSmemBytes, stream>>>(p, units, nUnits, next);
    return cudaGetLastError();
}

cudaError_t LaunchAggTaskCount(const AggTable *tables, int32_t nTasks, const TaskChunk *chunks, int32_t nChunks,
    int32_t keyKind, uint32_t *counts, cudaStream_t stream)
{
    if (nTasks <= 0) {
        return cudaSuccess;
    }
    const cudaError_t err = cudaMemsetAsync(counts, 0, sizeof(uint32_t) * nTasks, stream);
    if (err != cudaSuccess) {
        return err;
    }
    const int grid = nChunks < NumSMs() * 8 ? nChunks : NumSMs() * 8;
    TaskCountKernel<<<grid, 256, 0, stream>>>(tables, chunks, nChunks, keyKind, counts);
    return cudaGetLastError();
}

cudaError_t LaunchAggTaskPad(const uint32_t *groups, int32_t nTasks, uint32_t *padded, cudaStream_t stream)
{
    if (nTasks <= 0) {
        return cudaSuccess;
    }
    TaskPadKernel<<<(nTasks + 255) / 256, 256, 0, stream>>>(groups, nTasks, padded);
    return cudaGetLastError();
}

cudaError_t LaunchAggTaskExtract(const AggExtract &e, const AggTable *tables, int32_t nTasks, const TaskChunk *chunks,
    int32_t nChunks, const int64_t *offsets, unsigned long long *cursor, cudaStream_t stream)
{
    if (nTasks <= 0) {
        return cudaSuccess;
    }
    const cudaError_t err =
        cudaMemcpyAsync(cursor, offsets, sizeof(int64_t) * nTasks, cudaMemcpyDeviceToDevice, stream);
    if (err != cudaSuccess) {
        return err;
    }
    const int grid = nChunks < NumSMs() * 8 ? nChunks : NumSMs() * 8;
    TaskExtractKernel<<<grid, 256, 0, stream>>>(e, tables, chunks, nChunks, cursor);
    return cudaGetLastError();
}

int32_t AggPartSmemSlots(int32_t smemStride)
{
    return static_cast<int32_t>(kPartSmemBytes / (static_cast<size_t>(smemStride) * sizeof(uint64_t)));
}

cudaError_t LaunchAggPartition(const AggLaunch &p, const PartArgs &a, cudaStream_t stream)
{
    if (p.nTiles <= 0) {
        return cudaSuccess;
    }
    const int grid = p.nTiles < NumSMs() * 4 ? p.nTiles : NumSMs() * 4;
    if (a.stable) {
        // Per-tile counts, their prefixes in tile order, the layout, then the ordered scatter.
        if (p.key.kind == KEY_SINGLE) {
            PartTileHistKernel<KEY_SINGLE><<<grid, 512, 0, stream>>>(p, a);
        } else {
            PartTileHistKernel<KEY_PACKED><<<grid, 512, 0, stream>>>(p, a);
        }
        PartTileScanKernel<<<1 << a.partBits, 1024, 0, stream>>>(a, p.nTiles);
        PartLayoutKernel<<<1, kMaxParts, 0, stream>>>(a);
        if (p.key.kind == KEY_SINGLE) {
            PartScatterStableKernel<KEY_SINGLE><<<grid, kScatterThreads, 0, stream>>>(p, a);
        } else {
            PartScatterStableKernel<KEY_PACKED><<<grid, kScatterThreads, 0, stream>>>(p, a);
        }
        return cudaGetLastError();
    }
    if (p.key.kind == KEY_SINGLE) {
        PartHistKernel<KEY_SINGLE><<<grid, kHistThreads, 0, stream>>>(p, a);
    } else {
        PartHistKernel<KEY_PACKED><<<grid, kHistThreads, 0, stream>>>(p, a);
    }
    PartLayoutKernel<<<1, kMaxParts, 0, stream>>>(a);
    if (p.key.kind == KEY_SINGLE) {
        PartScatterKernel<KEY_SINGLE><<<grid, kScatterThreads, 0, stream>>>(p, a);
    } else {
        PartScatterKernel<KEY_PACKED><<<grid, kScatterThreads, 0, stream>>>(p, a);
    }
    return cudaGetLastError();
}

cudaError_t LaunchAggSketch(const AggLaunch &p, int32_t nSample, unsigned long long *tabKeys,
    unsigned int *tabCounts, unsigned long long *stats, cudaStream_t stream)
{
    if (p.nTiles <= 0 || nSample <= 0) {
        return cudaSuccess;
    }
    SketchInitKernel<<<64, 256, 0, stream>>>(tabKeys, tabCounts, stats);
    const int blocks = (nSample + 255) / 256;
    if (p.key.kind == KEY_SINGLE) {
        SketchKernel<KEY_SINGLE><<<blocks, 256, 0, stream>>>(p, nSample, tabKeys, tabCounts, stats);
    } else {
        SketchKernel<KEY_PACKED><<<blocks, 256, 0, stream>>>(p, nSample, tabKeys, tabCounts, stats);
    }
    SketchStatsKernel<<<64, 256, 0, stream>>>(tabKeys, tabCounts, stats);
    return cudaGetLastError();
}

// One CTA's registers in shared memory, merged into the global ones with atomicMax.
template <int kKind>
__global__ void __launch_bounds__(512) HllKernel(const __grid_constant__ AggLaunch p, unsigned int *regs)
{
    __shared__ unsigned int r[kHllRegs + 2];
    for (int i = threadIdx.x; i < kHllRegs + 2; i += blockDim.x) {
        r[i] = 0;
    }
    __syncthreads();
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        const TileDesc tile = p.tiles[t];
        const BatchDesc &b = p.batches[tile.batch];
        for (int row = threadIdx.x; row < tile.rows; row += blockDim.x) {
            const RowKey k = ReadKey(p.key, b, static_cast<int64_t>(tile.row0) + row, kKind);
            if (k.special >= 0) {
                r[kHllRegs + k.special] = 1u;
                continue;
            }
            const uint64_t h = Mix64(k.hash ^ 0x5851f42d4c957f2dull);  // bits independent of the table's
            const unsigned int reg = static_cast<unsigned int>(h >> (64 - kHllBits));
            const uint64_t rest = (h << kHllBits) | (1ull << (kHllBits - 1));
            atomicMax(&r[reg], static_cast<unsigned int>(__clzll(static_cast<long long>(rest)) + 1));
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kHllRegs + 2; i += blockDim.x) {
        if (r[i] != 0) {
            atomicMax(&regs[i], r[i]);
        }
    }
}

cudaError_t LaunchAggHll(const AggLaunch &p, unsigned int *regs, cudaStream_t stream)
{
    cudaError_t err = cudaMemsetAsync(regs, 0, (kHllRegs + 2) * sizeof(unsigned int), stream);
    if (err != cudaSuccess || p.nTiles <= 0) {
        return err;
    }
    const int grid = p.nTiles < DeviceSMCount() * 2 ? p.nTiles : DeviceSMCount() * 2;
    if (p.key.kind == KEY_SINGLE) {
        HllKernel<KEY_SINGLE><<<grid, 512, 0, stream>>>(p, regs);
    } else {
        HllKernel<KEY_PACKED><<<grid, 512, 0, stream>>>(p, regs);
    }
    return cudaGetLastError();
}

cudaError_t LaunchAlignColumn(const BatchDesc *batches, const TileDesc *tiles, int32_t nTiles,
    const int64_t *tileOutRow, const AlignCol &c, void *out, uint8_t *outNulls, cudaStream_t stream)
{
    if (nTiles <= 0) {
        return cudaSuccess;
    }
    const int grid = nTiles < DeviceSMCount() * 8 ? nTiles : DeviceSMCount() * 8;
    AlignColumnKernel<<<grid, 256, 0, stream>>>(batches, tiles, nTiles, tileOutRow, c, out, outNulls);
    return cudaGetLastError();
}

}  // namespace omg
