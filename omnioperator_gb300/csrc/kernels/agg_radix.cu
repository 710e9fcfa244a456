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

// Records rec + j * stepBytes.
struct RecRows {
    const RecLayout &l;
    const char *rec;
    int64_t stepBytes;
    __device__ __forceinline__ const char *At(int input, int, int j) const { return rec + j * stepBytes + l.off[input]; }
    __device__ __forceinline__ bool Nullable(int input) const { return l.nullOff[input] >= 0; }
    template <int N> __device__ __forceinline__ uint32_t Nulls(int input, uint32_t use) const
    {
        unsigned char byte[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            byte[j] = ((use >> j) & 1u) != 0
                ? __ldg(reinterpret_cast<const unsigned char *>(rec + j * stepBytes + l.nullOff[input]))
                : static_cast<unsigned char>(0);
        }
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            m |= (byte[j] != 0 ? 1u : 0u) << j;
        }
        return m;
    }
};

__device__ __forceinline__ unsigned int FinePart(uint64_t hash)
{
    return static_cast<unsigned int>(hash >> kRadixShift) & (kRadixFineParts - 1);
}

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
// store request too.
constexpr int kScatterThreads = 512;
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
constexpr int kSrcBatch = 6;

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
// Two 512-thread CTAs per SM, so that one's barriers and loads are under the other's work, take a unit
// each in steps of up to 2048 rows.  An atomic per row and accumulator was what bounded this: 64-bit adds
// and double sums in shared memory are compare-and-swap loops (1400 instructions a row where a group
// is hot), and FP64 additions are scarce.  So a step first sorts its rows by slot: a row takes its rank
// from the slot's counter (a native 32-bit atomic), the counters are scanned, and each input's values
// are exchanged into slot order through shared memory (gathered in slot order from the records, they
// took a request to L2 each).  Each thread then adds up four consecutive rows in registers and writes a
// group's sum once; a group that lies wholly in one thread's rows needs no atomic at all.
// The groups' slots are dense and found through an index of 32-bit words (a tag and a slot number) that
// is at most half full, so probe chains are short and a finished table is one copy.
constexpr int kRadixThreads = 512;
constexpr int kRadixRows = 4;  // rows per thread per step
constexpr int kStepRows = kRadixThreads * kRadixRows;
constexpr size_t kRadixSmemBytes = 112 * 1024;  // two CTAs per SM

// A step: its records, where the thread's own rows (row k * kRadixThreads + threadIdx.x of the step) go in slot
// order, and the exchange buffers.
struct Step {
    RecRows own;
    uint32_t placed;             // bit k: own row k has a place
    uint32_t pos[kRadixRows];
    uint64_t *values;            // [kStepRows]
    unsigned char *nulls;        // [kStepRows]
};

// A thread's rows in slot order.
struct Run {
    const char *step;      // the step's first record
    int32_t recBytes;
    uint32_t e[kRadixRows];  // slot << 16 | row of the step
    uint32_t live;         // bit j: row j exists
    uint32_t ends;         // bit j: row j is the last of its group here
    bool left, right;      // the first / last group goes on in a neighbouring thread's rows
    bool uniform;          // all rows of the warp are one group's
    __device__ __forceinline__ const char *Rec(int j) const { return step + (e[j] & 0xffffu) * recBytes; }
    __device__ __forceinline__ int Slot(int j) const { return static_cast<int>(e[j] >> 16); }
};

template <class T, class Op> __device__ __forceinline__ T WarpReduce(T v, Op op)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    return v;
}

// Combine the values x[j] of each group's rows (bit j of `use`) and store(slot, value, shared) each
// group's result once; shared: other threads store to the slot in this step too.
template <class T, class Op, class Store>
__device__ __forceinline__ void ForGroups(const Run &run, const T (&x)[kRadixRows], uint32_t use, T identity, Op op,
    Store store)
{
    if (run.uniform) {
        T v = identity;
#pragma unroll
        for (int j = 0; j < kRadixRows; ++j) {
            v = ((use >> j) & 1u) != 0 ? op(v, x[j]) : v;
        }
        v = WarpReduce(v, op);
        if (__any_sync(0xffffffffu, use != 0) && (threadIdx.x & 31) == 0) {
            store(run.Slot(0), v, true);
        }
        return;
    }
    T v = identity;
    bool any = false;
    bool shared = run.left;
#pragma unroll
    for (int j = 0; j < kRadixRows; ++j) {
        if ((use >> j) & 1u) {
            v = op(v, x[j]);
            any = true;
        }
        if ((run.ends >> j) & 1u) {
            if (any) {
                store(run.Slot(j), v, shared || (run.right && (run.live >> j) == 1u));
            }
            v = identity;
            any = false;
            shared = false;
        }
    }
}

__device__ __forceinline__ void MinWord(uint64_t *w, int64_t v, bool shared)
{
    if (shared) {
        AtomicMinI64(w, v);
    } else if (v < static_cast<int64_t>(*w)) {
        *w = static_cast<uint64_t>(v);
    }
}

__device__ __forceinline__ void MaxWord(uint64_t *w, int64_t v, bool shared)
{
    if (shared) {
        AtomicMaxI64(w, v);
    } else if (v > static_cast<int64_t>(*w)) {
        *w = static_cast<uint64_t>(v);
    }
}

__device__ __forceinline__ void AddWord(uint64_t *w, uint64_t v, bool shared)
{
    if (shared) {
        Red(w, v);
    } else {
        *w += v;
    }
}

__device__ __forceinline__ void ApplyInt(const AccSpec &s, const Run &run, const uint64_t (&bits)[kRadixRows],
    uint32_t use, uint64_t *st, int sw)
{
    long long x[kRadixRows];
#pragma unroll
    for (int j = 0; j < kRadixRows; ++j) {
        x[j] = SignExtend(bits[j], s.inWidth);
    }
    uint64_t *base = st + s.word;
    if (s.kind == ACC_ISUM) {
        ForGroups(run, x, use, 0ll, [](long long a, long long b) {
                return static_cast<long long>(static_cast<unsigned long long>(a) + static_cast<unsigned long long>(b)); },
            [&](int slot, long long v, bool shared) { AddWord(base + slot * sw, static_cast<uint64_t>(v), shared); });
    } else if (s.kind == ACC_WSUM2) {
        // Positive and negative magnitudes apart.  Up to 128 of less than 2^55 add up in one word, whose
        // halves go to the chunk sums; larger values go one by one.
        bool large = false;
#pragma unroll
        for (int j = 0; j < kRadixRows; ++j) {
            large = large || (((use >> j) & 1u) != 0 && (x[j] >= (1ll << 55) || x[j] <= -(1ll << 55)));
        }
        if (__any_sync(0xffffffffu, large)) {
#pragma unroll
            for (int j = 0; j < kRadixRows; ++j) {
                if ((use >> j) & 1u) {
                    const uint64_t m = x[j] >= 0 ? static_cast<uint64_t>(x[j]) : 0ull - static_cast<uint64_t>(x[j]);
                    uint64_t *w = base + run.Slot(j) * sw + (x[j] >= 0 ? 0 : 2);
                    Red(w, m & 0xffffffffull);
                    Red(w + 1, m >> 32);
                }
            }
            return;
        }
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            uint32_t mine = 0;
            unsigned long long m[kRadixRows];
#pragma unroll
            for (int j = 0; j < kRadixRows; ++j) {
                mine |= (x[j] < 0) == (side == 1) ? use & (1u << j) : 0u;
                m[j] = static_cast<unsigned long long>(side == 1 ? -x[j] : x[j]);
            }
            ForGroups(run, m, mine, 0ull, [](unsigned long long a, unsigned long long b) { return a + b; },
                [&](int slot, unsigned long long v, bool shared) {
                    uint64_t *w = base + slot * sw + 2 * side;
                    AddWord(w, v & 0xffffffffull, shared);
                    if ((v >> 32) != 0) {
                        AddWord(w + 1, v >> 32, shared);
                    }
                });
        }
    } else if (s.kind == ACC_IMIN) {
        ForGroups(run, x, use, static_cast<long long>(s.init), [](long long a, long long b) { return min(a, b); },
            [&](int slot, long long v, bool shared) { MinWord(base + slot * sw, v, shared); });
    } else {
        ForGroups(run, x, use, static_cast<long long>(s.init), [](long long a, long long b) { return max(a, b); },
            [&](int slot, long long v, bool shared) { MaxWord(base + slot * sw, v, shared); });
    }
}

// A decimal128 value into an exact sum or a min / max.
__device__ __forceinline__ void ApplyWide(const AccSpec &s, const char *at, uint64_t *w)
{
    const unsigned long long *v = reinterpret_cast<const unsigned long long *>(at);
    uint64_t lo = __ldg(v);
    uint64_t hi = __ldg(v + 1);
    if (s.kind != ACC_WSUM3) {
        AtomicMinMax128(w, lo, hi, s.kind == ACC_XMIN);
        return;
    }
    if (static_cast<int64_t>(hi) < 0) {  // magnitude = -(hi:lo)
        lo = ~lo + 1;
        hi = ~hi + (lo == 0 ? 1u : 0u);
        w += 4;
    }
    Red(w, lo & 0xffffffffull);
    Red(w + 1, lo >> 32);
    Red(w + 2, hi & 0xffffffffull);
    Red(w + 3, hi >> 32);
}

// Add x to the compensated sum at w (AtomicAddCompensated without the atomics).  A sum of at most
// 8 + 5 plain additions (a thread's rows, a warp's threads) comes in; every one after that is
// compensated.
__device__ __forceinline__ void AddDouble(uint64_t *w, double x, bool shared)
{
    if (shared) {
        AtomicAddCompensated(w, x, 0.0);
        return;
    }
    double *d = reinterpret_cast<double *>(w);
    const double old = d[0];
    if (__double_as_longlong(old) == 0) {  // the slot's first values
        d[0] = x;
        return;
    }
    const double sum = __dadd_rn(old, x);
    d[0] = sum;
    if (isfinite(sum)) {
        const double bv = __dsub_rn(sum, old);
        const double av = __dsub_rn(sum, bv);
        d[1] = __dadd_rn(d[1], __dadd_rn(__dsub_rn(old, av), __dsub_rn(x, bv)));
    }
}

// Input `input` of the thread's rows in slot order: its values (up to 8 bytes) and the rows whose value is
// not NULL.  Called by the whole CTA.
__device__ __forceinline__ uint32_t Exchange(const RecLayout &l, const Step &step, const Run &run, int input,
    int width, uint64_t (&bits)[kRadixRows])
{
    const bool nullable = l.nullOff[input] >= 0;
    uint64_t raw[kRadixRows];
    uint32_t null = 0;
    if (width > 0) {
        LoadBitsRows<kRadixRows>([&](int k) { return step.own.At(input, width, k); }, width, step.placed, raw);
    }
    if (nullable) {
        null = step.own.Nulls<kRadixRows>(input, step.placed);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRadixRows; ++k) {
        if ((step.placed >> k) & 1u) {
            if (width > 0) {
                step.values[step.pos[k]] = raw[k];
            }
            if (nullable) {
                step.nulls[step.pos[k]] = static_cast<unsigned char>((null >> k) & 1u);
            }
        }
    }
    __syncthreads();
    uint32_t use = run.live;
    if (nullable) {
        const uint32_t m = reinterpret_cast<const uint32_t *>(step.nulls)[threadIdx.x];
#pragma unroll
        for (int j = 0; j < kRadixRows; ++j) {
            use &= ~(((m >> (8 * j)) & 1u) << j);
        }
    }
    if (width > 0) {
#pragma unroll
        for (int j = 0; j < kRadixRows; j += 2) {
            const ulonglong2 v =
                *reinterpret_cast<const ulonglong2 *>(step.values + threadIdx.x * kRadixRows + j);
            bits[j] = v.x;
            bits[j + 1] = v.y;
        }
    }
    return use;
}

// Apply every accumulator but COUNT_ALL (counted with the sort) to the thread's rows.  Called by the whole
// CTA.
__device__ __forceinline__ void ApplyRun(const AggLaunch &p, const RecLayout &l, const Step &step, const Run &run,
    uint64_t *st)
{
    static_assert(kRadixRows == 4, "a thread's NULL bytes are read as one word");
    const int sw = p.table.slotWords;
    int input = -1;
    uint64_t bits[kRadixRows];
    uint32_t known = 0;  // the rows whose value is not NULL
    for (int a = 0; a < p.nAccs; ++a) {
        const AccSpec s = p.accs[a];
        if (s.kind == ACC_COUNT_ALL || (s.kind == ACC_NULLS && l.nullOff[s.input] < 0)) {
            continue;
        }
        if (s.input != input) {
            input = s.input;
            known = Exchange(l, step, run, input, l.width[input], bits);
        }
        const uint32_t use = known;
        uint64_t *base = st + s.word;
        switch (s.kind) {
            case ACC_NULLS: {
                const uint32_t count = run.live & ~use;
                if (!__any_sync(0xffffffffu, count != 0)) {
                    break;
                }
                unsigned int one[kRadixRows];
#pragma unroll
                for (int j = 0; j < kRadixRows; ++j) {
                    one[j] = 1u;
                }
                ForGroups(run, one, count, 0u, [](unsigned int x, unsigned int y) { return x + y; },
                    [&](int slot, unsigned int v, bool shared) {
                        // A shared table counts the rows of one unit (< 2^32): the word's low half.
                        unsigned int *w = LowHalf(base + slot * sw);
                        if (shared) {
                            atomicAdd(w, v);
                        } else {
                            *w += v;
                        }
                    });
                break;
            }
            case ACC_ISUM:
            case ACC_WSUM2:
            case ACC_IMIN:
            case ACC_IMAX:
                ApplyInt(s, run, bits, use, st, sw);
                break;
            case ACC_DSUM: {
                double x[kRadixRows];
#pragma unroll
                for (int j = 0; j < kRadixRows; ++j) {
                    x[j] = AsDouble(bits[j], s.inKind, s.inWidth);
                }
                // -0.0 + x is x for every x, so a single value passes through unchanged.
                ForGroups(run, x, use, -0.0, [](double u, double v) { return __dadd_rn(u, v); },
                    [&](int slot, double v, bool shared) { AddDouble(base + slot * sw, v, shared); });
                break;
            }
            case ACC_DMIN:
            case ACC_DMAX: {
                long long x[kRadixRows];
                uint32_t number = use;
#pragma unroll
                for (int j = 0; j < kRadixRows; ++j) {
                    const double d = AsDouble(bits[j], s.inKind, s.inWidth);
                    number &= ~((isnan(d) ? 1u : 0u) << j);
                    x[j] = OrderedFromDouble(d);
                }
                if (s.kind == ACC_DMIN) {
                    ForGroups(run, x, number, static_cast<long long>(s.init),
                        [](long long u, long long v) { return min(u, v); },
                        [&](int slot, long long v, bool shared) { MinWord(base + slot * sw, v, shared); });
                } else {
                    ForGroups(run, x, number, static_cast<long long>(s.init),
                        [](long long u, long long v) { return max(u, v); },
                        [&](int slot, long long v, bool shared) { MaxWord(base + slot * sw, v, shared); });
                }
                break;
            }
            default:  // decimal128 and string states: one row at a time
#pragma unroll
                for (int j = 0; j < kRadixRows; ++j) {
                    if (((use >> j) & 1u) == 0) {
                        continue;
                    }
                    uint64_t *w = base + run.Slot(j) * sw;
                    if (s.kind == ACC_SMIN || s.kind == ACC_SMAX) {
                        AtomicStrMinMax(p, s.input, w, SignExtend(bits[j], 4), s.kind == ACC_SMIN);
                    } else {
                        ApplyWide(s, run.Rec(j) + l.off[input], w);
                    }
                }
                break;
        }
    }
}

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

// Exclusive scan of cnt[0, n) in place, by the whole CTA; returns the total.  Each slot's count is added
// to the low half of its word `count` (a shared table counts the rows of one unit, < 2^32).
__device__ __forceinline__ unsigned int ScanCounts(unsigned int *cnt, int n, uint64_t *count, int sw,
    unsigned int *warpSums)
{
    constexpr int kWarps = kRadixThreads / 32;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int per = (n + kRadixThreads - 1) / kRadixThreads;
    const int first = threadIdx.x * per;
    unsigned int mine = 0;
    for (int i = 0; i < per; ++i) {
        mine += first + i < n ? cnt[first + i] : 0u;
    }
    unsigned int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y = __shfl_up_sync(0xffffffffu, inc, o);
        inc += lane >= o ? y : 0u;
    }
    if (lane == 31) {
        warpSums[warp] = inc;
    }
    __syncthreads();
    const unsigned int sums = lane < kWarps ? warpSums[lane] : 0u;
    const unsigned int total = __reduce_add_sync(0xffffffffu, sums);
    unsigned int run = __reduce_add_sync(0xffffffffu, lane < warp ? sums : 0u) + inc - mine;
    for (int i = 0; i < per; ++i) {
        if (first + i < n) {
            const unsigned int c = cnt[first + i];
            cnt[first + i] = run;
            run += c;
            *LowHalf(count + static_cast<int64_t>(first + i) * sw) += c;
        }
    }
    __syncthreads();
    return total;
}

template <int kKind>
__global__ void __launch_bounds__(kRadixThreads, 2) RadixAggKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ RecLayout l, const __grid_constant__ RadixAgg a, const __grid_constant__ SpillArgs sp)
{
    // The slots (the special ones first), the step's rows in slot order, the exchange buffers, the index, the
    // counters.
    extern __shared__ __align__(16) uint64_t smem[];
    __shared__ unsigned int newGroups;
    __shared__ unsigned int unitIndex;
    __shared__ unsigned int used;
    __shared__ unsigned int warpSums[kRadixThreads / 32];
    __shared__ unsigned long long denseBase;
    const int sw = p.table.slotWords;
    const int kw = p.table.keyWords;
    const unsigned int nSlots = static_cast<unsigned int>(p.smemSlots);
    const int nAll = static_cast<int>(nSlots) + kSpecialSlots;
    uint64_t *st = smem + kw;  // state words of slot i start at st + i * sw
    uint32_t *order = reinterpret_cast<uint32_t *>(smem + ((static_cast<int64_t>(nAll) * sw + 1) & ~int64_t(1)));
    uint64_t *values = reinterpret_cast<uint64_t *>(order + kStepRows);
    unsigned char *nulls = reinterpret_cast<unsigned char *>(values + kStepRows);
    unsigned int *index = reinterpret_cast<unsigned int *>(nulls + kStepRows);
    unsigned int *cnt = index + a.indexSize;
    const unsigned int indexMask = static_cast<unsigned int>(a.indexSize) - 1u;
    for (int i = threadIdx.x; i < nAll; i += kRadixThreads) {
        InitSlot(p, smem + static_cast<int64_t>(i) * sw);
        cnt[i] = 0;
    }
    for (int i = threadIdx.x; i < a.indexSize; i += kRadixThreads) {
        index[i] = 0;
    }
    if (threadIdx.x == 0) {
        newGroups = 0;
        used = 0;
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
                const uint32_t rows = min(stepRows, unit.rows - r0);
                Run run;
                run.step = RecAt(l, a.records, static_cast<uint64_t>(unit.first) + r0);
                run.recBytes = l.words * 8;
                uint32_t at[kRadixRows];  // slot << 16 | rank, or none
                Step step{RecRows{l, run.step + static_cast<int64_t>(threadIdx.x) * run.recBytes,
                              static_cast<int64_t>(kRadixThreads) * run.recBytes},
                    0, {}, values, nulls};
                constexpr int kBatch = 2;  // rows whose key loads are in flight together
#pragma unroll
                for (int k0 = 0; k0 < kRadixRows; k0 += kBatch) {
                    RowKey key[kBatch];
                    uint32_t use = 0;
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        use |= (k0 + k) * kRadixThreads + threadIdx.x < rows ? 1u << k : 0u;
                    }
                    ReadKeys<kKind, kBatch>(p.key,
                        RecRows{l, run.step + static_cast<int64_t>(k0 * kRadixThreads + threadIdx.x) * run.recBytes,
                            static_cast<int64_t>(kRadixThreads) * run.recBytes},
                        use, key);
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        at[k0 + k] = 0xffffffffu;
                        const uint32_t r = (k0 + k) * kRadixThreads + threadIdx.x;
                        if (r >= rows) {
                            continue;
                        }
                        int i = -3;
                        if (key[k].special >= 0) {
                            i = pass == 0 ? key[k].special : -3;
                        } else if (((key[k].hash >> (kRadixShift - kRadixMaxPassBits)) & passMask) == pass) {
                            i = FindGroup(smem, index, indexMask, &used, nSlots, sw, p.key, key[k], kKind);
                        }
                        if (i >= 0) {
                            at[k0 + k] = (static_cast<uint32_t>(i) << 16) | atomicAdd(&cnt[i], 1u);
                        } else if (i == -1) {
                            GlobalRecord(p, l, a.records, static_cast<uint64_t>(unit.first) + r0 + r, key[k], kKind,
                                &newGroups);
                        } else if (i == -2) {
                            SetError(p.error, 7);
                        }
                    }
                }
                __syncthreads();
                const int nUsed = static_cast<int>(min(used, nSlots)) + kSpecialSlots;
                const int total = static_cast<int>(ScanCounts(cnt, nUsed, st + p.accs[0].word, sw, warpSums));
#pragma unroll
                for (int k = 0; k < kRadixRows; ++k) {
                    if (at[k] != 0xffffffffu) {
                        step.placed |= 1u << k;
                        step.pos[k] = cnt[at[k] >> 16] + (at[k] & 0xffffu);
                        order[step.pos[k]] =
                            (at[k] & 0xffff0000u) | static_cast<uint32_t>(k * kRadixThreads + threadIdx.x);
                    }
                }
                __syncthreads();
                for (int i = threadIdx.x; i < nUsed; i += kRadixThreads) {
                    cnt[i] = 0;
                }
                const int pos = threadIdx.x * kRadixRows;
                const int n = min(max(total - pos, 0), kRadixRows);
#pragma unroll
                for (int j = 0; j < kRadixRows; j += 4) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(order + pos + j);
                    run.e[j] = v.x;
                    run.e[j + 1] = v.y;
                    run.e[j + 2] = v.z;
                    run.e[j + 3] = v.w;
                }
                run.live = (1u << n) - 1u;
                run.left = n > 0 && pos > 0 && (order[pos - 1] >> 16) == (run.e[0] >> 16);
                const uint32_t next = pos + kRadixRows < total ? order[pos + kRadixRows] >> 16 : 0xffffffffu;
                run.right = n == kRadixRows && next == (run.e[kRadixRows - 1] >> 16);
                run.ends = 0;
#pragma unroll
                for (int j = 0; j < kRadixRows; ++j) {
                    const bool last = j == n - 1 || (j + 1 < kRadixRows && j + 1 < n &&
                        (run.e[j] >> 16) != (run.e[(j + 1) % kRadixRows] >> 16));
                    run.ends |= last ? 1u << j : 0u;
                }
                const uint32_t slot0 = __shfl_sync(0xffffffffu, run.e[0] >> 16, 0);
                run.uniform = __all_sync(0xffffffffu,
                    run.ends == 1u << (kRadixRows - 1) && (run.e[0] >> 16) == slot0) != 0;
                ApplyRun(p, l, step, run, st);
                __syncthreads();
            }
            const unsigned int groups = min(used, nSlots);
            if (threadIdx.x < kSpecialSlots) {
                const int s = threadIdx.x;
                uint64_t *slot = smem + static_cast<int64_t>(s) * sw;
                if (slot[kw + p.accs[0].word] != 0) {
                    atomicExch(&p.table.specialUsed[s], 1u);
                    MergeStates(p, p.accs, p.nAccs, slot + kw, p.table.slots + (p.table.capacity + s) * sw + kw);
                    InitSlot(p, slot);
                }
            }
            uint64_t *first = smem + static_cast<int64_t>(kSpecialSlots) * sw;
            if (unit.multi != 0) {
                for (unsigned int i = threadIdx.x; i < groups; i += kRadixThreads) {
                    MergeRecord<kKind>(p, sp, first + static_cast<int64_t>(i) * sw, &newGroups);
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
                    for (unsigned int w = threadIdx.x; w < groups * sw; w += kRadixThreads) {
                        dst[w] = first[w];
                    }
                }
            }
            __syncthreads();
            for (unsigned int i = threadIdx.x; i < groups; i += kRadixThreads) {
                InitSlot(p, first + static_cast<int64_t>(i) * sw);
            }
            for (int i = threadIdx.x; i < a.indexSize; i += kRadixThreads) {
                index[i] = 0;
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

int32_t AggRadixSlots(int32_t slotWords, int32_t *indexSize)
{
    // The most slots that fit beside an index of at least twice as many words.
    const int64_t perSlot = static_cast<int64_t>(slotWords) * 8 + 4;
    int32_t best = 0;
    for (int32_t size = 256; size <= 16384; size *= 2) {
        const int64_t room = static_cast<int64_t>(kRadixSmemBytes) - kStepRows * (4 + 8 + 1) - size * 4 - 16;
        const int64_t n = room / perSlot - kSpecialSlots;
        const int32_t slots = static_cast<int32_t>(n < size / 2 ? n : size / 2);
        if (slots > best) {
            best = slots;
            *indexSize = size;
        }
    }
    return best;
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
    kernel<<<grid, kRadixThreads, kRadixSmemBytes, stream>>>(p, l, a, sp);
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
