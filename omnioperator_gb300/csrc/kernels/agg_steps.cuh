// Aggregation of rows by one CTA in steps, in shared memory.
//
// A step is up to 2048 rows of one batch or one run of records.  An atomic per row and accumulator was
// what bounded shared tables: 64-bit adds and double sums in shared memory are compare-and-swap loops
// (1400 instructions a row where a group is hot), and FP64 additions are scarce.  So a step first sorts
// its rows by slot: a row takes its rank from the slot's counter (a native 32-bit atomic), the counters
// are scanned, and each input's values are exchanged into slot order through shared memory (gathered
// in slot order from the rows, they took a request to L2 each).  Each thread then adds up four
// consecutive rows in registers and writes a group's sum once; a group that lies wholly in one
// thread's rows needs no atomic at all.
#pragma once

#include "agg_device.cuh"

namespace omg {
namespace {

constexpr int kStepThreads = 512;
constexpr int kStepThreadRows = 4;  // rows per thread per step
constexpr int kStepRows = kStepThreads * kStepThreadRows;

// Where the thread's own rows (row k * kStepThreads + threadIdx.x of the step) go in slot order, and the
// exchange buffers.
struct Step {
    uint32_t placed;             // bit k: own row k has a place
    uint32_t pos[kStepThreadRows];
    uint64_t *values;            // [kStepRows]
    unsigned char *nulls;        // [kStepRows]
};

// A thread's rows in slot order.
struct Run {
    uint32_t e[kStepThreadRows];  // slot << 16 | row of the step
    uint32_t live;         // bit j: row j exists
    uint32_t ends;         // bit j: row j is the last of its group here
    bool left, right;      // the first / last group goes on in a neighbouring thread's rows
    bool uniform;          // all rows of the warp are one group's
    __device__ __forceinline__ uint32_t Row(int j) const { return e[j] & 0xffffu; }
    __device__ __forceinline__ int Slot(int j) const { return static_cast<int>(e[j] >> 16); }
};

// The thread's own rows k0 + j of the step, as ReadKeys and LoadBitsRows take them.
template <class Rows> struct OwnRows {
    const Rows &rows;
    int k0;
    __device__ __forceinline__ uint32_t R(int j) const { return (k0 + j) * kStepThreads + threadIdx.x; }
    __device__ __forceinline__ const char *At(int input, int width, int j) const { return rows.RowAt(input, width, R(j)); }
    __device__ __forceinline__ bool Nullable(int input) const { return rows.Nullable(input); }
    template <int N> __device__ __forceinline__ uint32_t Nulls(int input, uint32_t use) const
    {
        uint32_t byte[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            byte[j] = ((use >> j) & 1u) != 0 ? rows.NullByte(input, R(j)) : 0u;
        }
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            m |= rows.NullBit(byte[j], R(j)) << j;
        }
        return m & use;
    }
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
__device__ __forceinline__ void ForGroups(const Run &run, const T (&x)[kStepThreadRows], uint32_t use, T identity, Op op,
    Store store)
{
    if (run.uniform) {
        T v = identity;
#pragma unroll
        for (int j = 0; j < kStepThreadRows; ++j) {
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
    for (int j = 0; j < kStepThreadRows; ++j) {
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

__device__ __forceinline__ void ApplyInt(const AccSpec &s, const Run &run, const uint64_t (&bits)[kStepThreadRows],
    uint32_t use, uint64_t *st, int sw)
{
    long long x[kStepThreadRows];
#pragma unroll
    for (int j = 0; j < kStepThreadRows; ++j) {
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
        for (int j = 0; j < kStepThreadRows; ++j) {
            large = large || (((use >> j) & 1u) != 0 && (x[j] >= (1ll << 55) || x[j] <= -(1ll << 55)));
        }
        if (__any_sync(0xffffffffu, large)) {
#pragma unroll
            for (int j = 0; j < kStepThreadRows; ++j) {
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
            unsigned long long m[kStepThreadRows];
#pragma unroll
            for (int j = 0; j < kStepThreadRows; ++j) {
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

// A sum of doubles and the rounding errors of its additions (NaN once the sum is not finite: AddDouble leaves
// them out then).
struct Sum {
    double sum;
    double err;
};

__device__ __forceinline__ bool IsZero(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ bool IsFinite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

__device__ __forceinline__ void AddTo(Sum &a, double x)
{
    const double next = __dadd_rn(a.sum, x);
    a.err = __dadd_rn(a.err, SumError(a.sum, x, next));
    a.sum = next;
}

// Add v to the compensated sum at w.  FP64 operations bound it (an SM does two a cycle, comparisons among them, and a
// warp goes through the shared and the unshared ones for each of its threads' rows), so both kinds of store take
// one way as far as they can, zeros are told by their bits, and nothing is compensated for on a slot's first value.
__device__ __forceinline__ void AddDouble(uint64_t *w, const Sum &v, bool shared)
{
    double *d = reinterpret_cast<double *>(w);
    const double old = shared ? atomicAdd(d, v.sum) : d[0];
    double sum = v.sum;
    double err = v.err;
    if (!IsZero(old) || IsZero(v.sum)) {  // 0.0 + -0.0 is 0.0
        sum = __dadd_rn(old, v.sum);
        err = __dadd_rn(err, SumError(old, v.sum, sum));
    }
    if (!shared) {
        d[0] = sum;
    }
    if (!IsZero(err) && IsFinite(sum)) {
        if (shared) {
            atomicAdd(d + 1, err);
        } else {
            d[1] = __dadd_rn(d[1], err);
        }
    }
}

// The sum over the warp's threads, in thread 0.  Each value is cut at a bit that is the same for all of them, so far
// below 2^8 times their largest power of two that the upper parts, 46 bits each, add up without rounding, and the
// lower parts' roundings are of second order: 14 FP64 operations where five times AddTo and an error takes 25
// (2^26 rows of a skewed two-column key, decimal sum, count and average: 9.60 -> 9.18 ms; 8.54 to 8.77 with plain
// sums in the runs).
__device__ __forceinline__ void SumWarp(Sum &v)
{
    const unsigned int most =
        __reduce_max_sync(0xffffffffu, static_cast<unsigned int>(__double2hiint(v.sum)) & 0x7ff00000u);
    if (most < (0x7ffu - 9u) << 20) {
        const double cut = __hiloint2double(static_cast<int>(most + (8u << 20)), 0);
        const double top = __dsub_rn(__dadd_rn(cut, v.sum), cut);
        v.err = __dadd_rn(v.err, __dsub_rn(v.sum, top));
        v.sum = top;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v.sum = __dadd_rn(v.sum, __shfl_down_sync(0xffffffffu, v.sum, o));
            v.err = __dadd_rn(v.err, __shfl_down_sync(0xffffffffu, v.err, o));
        }
        return;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {  // near the largest double, infinite, or not a number
        const double sum = __shfl_down_sync(0xffffffffu, v.sum, o);
        const double err = __shfl_down_sync(0xffffffffu, v.err, o);
        AddTo(v, sum);
        v.err = __dadd_rn(v.err, err);
    }
}

// ForGroups for sums of doubles into the states at base.  A run's first value needs no addition.
__device__ __forceinline__ void SumGroups(const Run &run, const double (&x)[kStepThreadRows], uint32_t use,
    uint64_t *base, int sw)
{
    Sum v{-0.0, 0.0};  // -0.0 + x is x for every x
    bool any = false;
    bool shared = run.left;
#pragma unroll
    for (int j = 0; j < kStepThreadRows; ++j) {
        if ((use >> j) & 1u) {
            if (any) {
                AddTo(v, x[j]);
            } else {
                v.sum = x[j];
            }
            any = true;
        }
        if (!run.uniform && ((run.ends >> j) & 1u) != 0) {
            if (any) {
                AddDouble(base + run.Slot(j) * sw, v, shared || (run.right && (run.live >> j) == 1u));
            }
            v = Sum{-0.0, 0.0};
            any = false;
            shared = false;
        }
    }
    if (run.uniform) {
        SumWarp(v);
        if (__any_sync(0xffffffffu, use != 0) && (threadIdx.x & 31) == 0) {
            AddDouble(base + run.Slot(0) * sw, v, true);
        }
    }
}

// Input `input` of the thread's rows in slot order: its values (up to 8 bytes) and the rows whose value is
// not NULL.  Called by the whole CTA.
template <class Rows>
__device__ __forceinline__ uint32_t Exchange(const Rows &rows, const Step &step, const Run &run, int input,
    uint64_t (&bits)[kStepThreadRows])
{
    const int width = rows.Width(input);
    const bool nullable = rows.Nullable(input);
    const OwnRows<Rows> own{rows, 0};
    uint64_t raw[kStepThreadRows];
    uint32_t null = 0;
    if (width > 0) {
        LoadBitsRows<kStepThreadRows>([&](int k) { return own.At(input, width, k); }, width, step.placed, raw);
    }
    if (nullable) {
        null = own.template Nulls<kStepThreadRows>(input, step.placed);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kStepThreadRows; ++k) {
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
        for (int j = 0; j < kStepThreadRows; ++j) {
            use &= ~(((m >> (8 * j)) & 1u) << j);
        }
    }
    if (width > 0) {
#pragma unroll
        for (int j = 0; j < kStepThreadRows; j += 2) {
            const ulonglong2 v =
                *reinterpret_cast<const ulonglong2 *>(step.values + threadIdx.x * kStepThreadRows + j);
            bits[j] = v.x;
            bits[j + 1] = v.y;
        }
    }
    return use;
}

// Apply every accumulator but COUNT_ALL (counted with the sort) to the thread's rows.  Called by the whole
// CTA.
template <class Rows>
__device__ __forceinline__ void ApplyRun(const AggLaunch &p, const Rows &rows, const Step &step, const Run &run,
    uint64_t *st)
{
    static_assert(kStepThreadRows == 4, "a thread's NULL bytes are read as one word");
    const int sw = p.smemStride;
    int input = -1;
    uint64_t bits[kStepThreadRows];
    uint32_t known = 0;  // the rows whose value is not NULL
    for (int a = 0; a < p.nAccs; ++a) {
        const AccSpec s = p.accs[a];
        if (s.kind == ACC_COUNT_ALL || (s.kind == ACC_NULLS && !rows.Nullable(s.input))) {
            continue;
        }
        if (s.input != input) {
            input = s.input;
            known = Exchange(rows, step, run, input, bits);
        }
        const uint32_t use = known;
        uint64_t *base = st + s.word;
        switch (s.kind) {
            case ACC_NULLS: {
                const uint32_t count = run.live & ~use;
                if (!__any_sync(0xffffffffu, count != 0)) {
                    break;
                }
                unsigned int one[kStepThreadRows];
#pragma unroll
                for (int j = 0; j < kStepThreadRows; ++j) {
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
                double x[kStepThreadRows];
#pragma unroll
                for (int j = 0; j < kStepThreadRows; ++j) {
                    x[j] = AsDouble(bits[j], s.inKind, s.inWidth);
                }
                SumGroups(run, x, use, base, sw);
                break;
            }
            case ACC_DMIN:
            case ACC_DMAX: {
                long long x[kStepThreadRows];
                uint32_t number = use;
#pragma unroll
                for (int j = 0; j < kStepThreadRows; ++j) {
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
                for (int j = 0; j < kStepThreadRows; ++j) {
                    if (((use >> j) & 1u) == 0) {
                        continue;
                    }
                    uint64_t *w = base + run.Slot(j) * sw;
                    if (s.kind == ACC_SMIN || s.kind == ACC_SMAX) {
                        AtomicStrMinMax(p, s.input, w, SignExtend(bits[j], 4), s.kind == ACC_SMIN);
                    } else {
                        ApplyWide(s, rows.RowAt(input, 16, run.Row(j)), w);
                    }
                }
                break;
        }
    }
}

// Exclusive scan of cnt[0, n) in place, by the whole CTA; returns the total.  Each slot's count is added
// to the low half of its word `count` (a shared table counts the rows of one unit, < 2^32).
__device__ __forceinline__ unsigned int ScanCounts(unsigned int *cnt, int n, uint64_t *count, int sw,
    unsigned int *warpSums)
{
    constexpr int kWarps = kStepThreads / 32;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int per = (n + kStepThreads - 1) / kStepThreads;
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

// The CTA's table and scratch in dynamic shared memory: the slots (the special ones first), the step's rows
// in slot order, the exchange buffers, the index, the counters.
struct StepTable {
    uint64_t *slots;
    uint64_t *st;  // state words of slot i start at st + i * smemStride
    uint32_t *order;
    uint64_t *values;
    unsigned char *nulls;
    unsigned int *index;
    unsigned int *cnt;
    int32_t indexSize;
    int32_t nAll;           // slots, the special ones among them
    unsigned int nSlots;    // groups
    unsigned int *used;     // groups taken (may pass nSlots)
    unsigned int *warpSums; // [kStepThreads / 32]
};

// Groups that a table in `smemBytes` of dynamic shared memory holds beside an index of at least twice as many
// words.
inline int32_t StepTableSlots(int32_t smemStride, size_t smemBytes, int32_t *indexSize)
{
    const int64_t perSlot = static_cast<int64_t>(smemStride) * 8 + 4;
    int32_t best = 0;
    for (int32_t size = 256; size <= 16384; size *= 2) {
        const int64_t room = static_cast<int64_t>(smemBytes) - kStepRows * (4 + 8 + 1) - size * 4 - 16;
        const int64_t n = room / perSlot - kSpecialSlots;
        const int32_t slots = static_cast<int32_t>(n < size / 2 ? n : size / 2);
        if (slots > best) {
            best = slots;
            *indexSize = size;
        }
    }
    return best;
}

__device__ __forceinline__ StepTable MakeStepTable(uint64_t *smem, int nAll, int sw, int kw, unsigned int nSlots,
    int32_t indexSize, unsigned int *used, unsigned int *warpSums)
{
    StepTable t;
    t.slots = smem;
    t.st = smem + kw;
    t.order = reinterpret_cast<uint32_t *>(smem + ((static_cast<int64_t>(nAll) * sw + 1) & ~int64_t(1)));
    t.values = reinterpret_cast<uint64_t *>(t.order + kStepRows);
    t.nulls = reinterpret_cast<unsigned char *>(t.values + kStepRows);
    t.index = reinterpret_cast<unsigned int *>(t.nulls + kStepRows);
    t.cnt = t.index + indexSize;
    t.indexSize = indexSize;
    t.nAll = nAll;
    t.nSlots = nSlots;
    t.used = used;
    t.warpSums = warpSums;
    return t;
}

__device__ __forceinline__ void InitStepTable(const AggLaunch &p, const StepTable &t)
{
    for (int i = threadIdx.x; i < t.nAll; i += kStepThreads) {
        InitSlot(p, t.slots + static_cast<int64_t>(i) * p.smemStride);
        t.cnt[i] = 0;
    }
    for (int i = threadIdx.x; i < t.indexSize; i += kStepThreads) {
        t.index[i] = 0;
    }
    if (threadIdx.x == 0) {
        *t.used = 0;
    }
}

// Rows [0, n) of `rows` (n <= kStepRows) into the table, by the whole CTA.  Rows whose key wants(key) rejects are
// left out; miss(r, key) takes row r when its group found no slot.
template <int kKind, class Rows, class Wants, class Miss>
__device__ __forceinline__ void AggregateStep(const AggLaunch &p, const Rows &rows, uint32_t n, const StepTable &t,
    Wants wants, Miss miss)
{
    const int sw = p.smemStride;
    Step step;
    step.placed = 0;
    step.values = t.values;
    step.nulls = t.nulls;
    uint32_t at[kStepThreadRows];  // slot << 16 | rank, or none
    constexpr int kBatch = 2;  // rows whose key loads are in flight together
#pragma unroll
    for (int k0 = 0; k0 < kStepThreadRows; k0 += kBatch) {
        RowKey key[kBatch];
        uint32_t use = 0;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            use |= (k0 + k) * kStepThreads + threadIdx.x < n ? 1u << k : 0u;
        }
        ReadKeys<kKind, kBatch>(p.key, OwnRows<Rows>{rows, k0}, use, key);
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            at[k0 + k] = 0xffffffffu;
            if (((use >> k) & 1u) == 0 || !wants(key[k])) {
                continue;
            }
            const int i = key[k].special >= 0
                ? key[k].special
                : FindGroup(t.slots, t.index, static_cast<unsigned int>(t.indexSize) - 1u, t.used, t.nSlots, sw, p.key,
                      key[k], kKind);
            if (i >= 0) {
                at[k0 + k] = (static_cast<uint32_t>(i) << 16) | atomicAdd(&t.cnt[i], 1u);
            } else if (i == -1) {
                miss((k0 + k) * kStepThreads + threadIdx.x, key[k]);
            } else {
                SetError(p.error, 7);
            }
        }
    }
    __syncthreads();
    const int nUsed = static_cast<int>(min(*t.used, t.nSlots)) + kSpecialSlots;
    const int total = static_cast<int>(ScanCounts(t.cnt, nUsed, t.st + p.accs[0].word, sw, t.warpSums));
#pragma unroll
    for (int k = 0; k < kStepThreadRows; ++k) {
        if (at[k] != 0xffffffffu) {
            step.placed |= 1u << k;
            step.pos[k] = t.cnt[at[k] >> 16] + (at[k] & 0xffffu);
            t.order[step.pos[k]] = (at[k] & 0xffff0000u) | static_cast<uint32_t>(k * kStepThreads + threadIdx.x);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nUsed; i += kStepThreads) {
        t.cnt[i] = 0;
    }
    Run run;
    const int pos = threadIdx.x * kStepThreadRows;
    const int mine = min(max(total - pos, 0), kStepThreadRows);
#pragma unroll
    for (int j = 0; j < kStepThreadRows; j += 4) {
        const uint4 v = *reinterpret_cast<const uint4 *>(t.order + pos + j);
        run.e[j] = v.x;
        run.e[j + 1] = v.y;
        run.e[j + 2] = v.z;
        run.e[j + 3] = v.w;
    }
    run.live = (1u << mine) - 1u;
    run.left = mine > 0 && pos > 0 && (t.order[pos - 1] >> 16) == (run.e[0] >> 16);
    const uint32_t next = pos + kStepThreadRows < total ? t.order[pos + kStepThreadRows] >> 16 : 0xffffffffu;
    run.right = mine == kStepThreadRows && next == (run.e[kStepThreadRows - 1] >> 16);
    run.ends = 0;
#pragma unroll
    for (int j = 0; j < kStepThreadRows; ++j) {
        const bool last = j == mine - 1 || (j + 1 < kStepThreadRows && j + 1 < mine &&
            (run.e[j] >> 16) != (run.e[(j + 1) % kStepThreadRows] >> 16));
        run.ends |= last ? 1u << j : 0u;
    }
    const uint32_t slot0 = __shfl_sync(0xffffffffu, run.e[0] >> 16, 0);
    run.uniform = __all_sync(0xffffffffu,
        run.ends == 1u << (kStepThreadRows - 1) && (run.e[0] >> 16) == slot0) != 0;
    ApplyRun(p, rows, step, run, t.st);
    __syncthreads();
}

}  // namespace
}  // namespace omg
