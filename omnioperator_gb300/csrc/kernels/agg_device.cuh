// Device functions of the hash aggregation kernels: row keys and inputs, state updates and merges,
// the global table and the shared-memory tables.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "plan.h"

namespace omg {
namespace {

constexpr int kSmemProbe = 8;
constexpr uint64_t kTagLocked = 1;

// ------------------------------------------------------------------ key handling
struct RowKey {
    uint64_t w[3];  // KEY_SINGLE: w[0] = key; KEY_PACKED: packed words
    uint64_t hash;
    int special;    // -1 normal, kNullSlotOffset / kSentinelSlotOffset for the special groups
};

__device__ __forceinline__ void OrKeyWord(RowKey &k, int i, uint64_t v)
{
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        k.w[j] |= j == i ? v : 0ull;
    }
}

__device__ __forceinline__ uint64_t KeyWordsHash(const RowKey &k, int words)
{
    uint64_t h = 0x9e3779b97f4a7c15ull;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        h = j < words ? Mix64(h ^ k.w[j]) : h;
    }
    return h;
}

// Where a row's inputs are read from: row `row` of a batch's columns.
struct BatchRow {
    const BatchDesc &b;
    int64_t row;
    __device__ __forceinline__ bool Null(int input) const { return NullRO(b.nulls[input], row); }
    __device__ __forceinline__ uint64_t Bits(int input, int width) const { return LoadBitsRO(b.cols[input], row, width); }
    __device__ __forceinline__ const uint64_t *Wide(int input) const
    {
        return static_cast<const uint64_t *>(b.cols[input]) + 2 * row;
    }
};

template <class Row> __device__ __forceinline__ RowKey ReadKeyOf(const KeySpec &ks, const Row &src, int kind)
{
    RowKey k;
    k.w[0] = k.w[1] = k.w[2] = 0;
    k.special = -1;
    if (kind == KEY_SINGLE) {
        const KeyCol &c = ks.cols[0];
        if (src.Null(c.input)) {
            k.special = kNullSlotOffset;
            k.hash = 0;
            return k;
        }
        uint64_t v = static_cast<uint64_t>(SignExtend(src.Bits(c.input, c.width), c.width));
        k.w[0] = v;
        if (v == kEmptyKey) {
            k.special = kSentinelSlotOffset;
        }
        k.hash = Mix64(v);
        return k;
    }
    // The loops are unrolled over constant word indices, so the words stay in registers.
    uint32_t mask = 0;
#pragma unroll
    for (int ci = 0; ci < kMaxKeyCols; ++ci) {
        if (ci >= ks.nCols) {
            break;
        }
        const KeyCol &c = ks.cols[ci];
        if (src.Null(c.input)) {
            mask |= 1u << ci;
            continue;
        }
        const int wi = c.byteOffset >> 3;
        const int sh = (c.byteOffset & 7) * 8;
        uint64_t lo, hi = 0;
        if (c.width == 16) {
            const uint64_t *p = src.Wide(c.input);
            lo = p[0];
            hi = p[1];
        } else {
            lo = src.Bits(c.input, c.width) << sh;
        }
        OrKeyWord(k, wi, lo);
        OrKeyWord(k, wi + 1, hi);
    }
    OrKeyWord(k, ks.maskByte >> 3, static_cast<uint64_t>(mask) << ((ks.maskByte & 7) * 8));
    k.hash = KeyWordsHash(k, ks.words);
    return k;
}

__device__ __forceinline__ RowKey ReadKey(const KeySpec &ks, const BatchDesc &b, int64_t row, int kind)
{
    return ReadKeyOf(ks, BatchRow{b, row}, kind);
}

// ---- several rows at once
// A load is only in flight with another row's if nothing between them waits for it or branches on it, so
// the loads of a value of N rows come first, under one branch on its width, and what uses them after.
// at(j): the address of row j's value; bit j of `use`: row j exists.
template <int N, class At>
__device__ __forceinline__ void LoadBitsRows(At at, int width, uint32_t use, uint64_t (&v)[N])
{
    switch (width) {
        case 1:
#pragma unroll
            for (int j = 0; j < N; ++j) {
                v[j] = ((use >> j) & 1u) != 0 ? __ldg(reinterpret_cast<const unsigned char *>(at(j))) : 0;
            }
            break;
        case 2:
#pragma unroll
            for (int j = 0; j < N; ++j) {
                v[j] = ((use >> j) & 1u) != 0 ? __ldg(reinterpret_cast<const unsigned short *>(at(j))) : 0;
            }
            break;
        case 4:
#pragma unroll
            for (int j = 0; j < N; ++j) {
                v[j] = ((use >> j) & 1u) != 0 ? __ldg(reinterpret_cast<const unsigned int *>(at(j))) : 0;
            }
            break;
        default:
#pragma unroll
            for (int j = 0; j < N; ++j) {
                v[j] = ((use >> j) & 1u) != 0 ? __ldg(reinterpret_cast<const unsigned long long *>(at(j))) : 0;
            }
            break;
    }
}

// Rows row0 + j * kStep of a batch.
template <int kStep> struct BatchRows {
    const BatchDesc &b;
    int64_t row0;
    __device__ __forceinline__ const char *At(int input, int width, int j) const
    {
        return static_cast<const char *>(b.cols[input]) + (row0 + j * kStep) * width;
    }
    __device__ __forceinline__ bool Nullable(int input) const { return b.nulls[input] != nullptr; }
    template <int N> __device__ __forceinline__ uint32_t Nulls(int input, uint32_t use) const
    {
        const unsigned char *nulls = reinterpret_cast<const unsigned char *>(b.nulls[input]);
        unsigned int byte[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            byte[j] = ((use >> j) & 1u) != 0 ? __ldg(nulls + ((row0 + j * kStep) >> 3)) : 0u;
        }
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            m |= ((byte[j] >> ((row0 + j * kStep) & 7)) & 1u) << j;
        }
        return m;
    }
};

// ReadKey of N rows (bit j of `use`; the others' keys are meaningless).
template <int kKind, int N, class Rows>
__device__ __forceinline__ void ReadKeys(const KeySpec &ks, const Rows &rows, uint32_t use, RowKey (&k)[N])
{
    if constexpr (kKind == KEY_SINGLE) {
        const KeyCol &c = ks.cols[0];
        uint64_t raw[N];
        LoadBitsRows<N>([&](int j) { return rows.At(c.input, c.width, j); }, c.width, use, raw);
        const uint32_t null = rows.Nullable(c.input) ? rows.template Nulls<N>(c.input, use) : 0u;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const uint64_t v = static_cast<uint64_t>(SignExtend(raw[j], c.width));
            const bool isNull = ((null >> j) & 1u) != 0;
            k[j].w[0] = isNull ? 0ull : v;
            k[j].w[1] = k[j].w[2] = 0;
            k[j].special = isNull ? kNullSlotOffset : (v == kEmptyKey ? kSentinelSlotOffset : -1);
            k[j].hash = isNull ? 0ull : Mix64(v);
        }
    } else {
        // Two columns at a time: both columns' loads are in flight together.
        uint32_t nulls[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
            k[j].w[0] = k[j].w[1] = k[j].w[2] = 0;
            k[j].special = -1;
            nulls[j] = 0;
        }
        for (int c0 = 0; c0 < ks.nCols; c0 += 2) {
            uint64_t raw[2][N];
            uint32_t null[2] = {0, 0};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (c0 + i < ks.nCols) {
                    const KeyCol &c = ks.cols[c0 + i];
                    LoadBitsRows<N>([&](int j) { return rows.At(c.input, c.width, j); }, c.width, use, raw[i]);
                    null[i] = rows.Nullable(c.input) ? rows.template Nulls<N>(c.input, use) : 0u;
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (c0 + i >= ks.nCols) {
                    break;
                }
                const KeyCol &c = ks.cols[c0 + i];
                const int wi = c.byteOffset >> 3;
                const int sh = (c.byteOffset & 7) * 8;
                if (c.width == 16) {
                    uint64_t hi[N];
                    LoadBitsRows<N>([&](int j) { return rows.At(c.input, c.width, j) + 8; }, 8, use & ~null[i], hi);
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        OrKeyWord(k[j], wi + 1, hi[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    const bool isNull = ((null[i] >> j) & 1u) != 0;
                    OrKeyWord(k[j], wi, isNull ? 0ull : raw[i][j] << sh);
                    nulls[j] |= (isNull ? 1u : 0u) << (c0 + i);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            OrKeyWord(k[j], ks.maskByte >> 3, static_cast<uint64_t>(nulls[j]) << ((ks.maskByte & 7) * 8));
            k[j].hash = KeyWordsHash(k[j], ks.words);
        }
    }
}

// Published tag of a packed slot: never 0 (free) or 1 (locked).
__device__ __forceinline__ uint64_t PublishedTag(uint64_t hash) { return (hash | 2ull) & ~1ull; }

// ------------------------------------------------------------------ row inputs
// A row's key plus the values and null bits of up to kRegInputs narrow inputs, all loaded up
// front through the read-only path so their latencies overlap.
struct RowIn {
    RowKey k;
    uint64_t v[kRegInputs];  // raw bits, zero-extended
    uint32_t nulls;          // bit i: register input i is NULL
};

template <int kKind>
__device__ __forceinline__ RowIn LoadRow(const AggLaunch &p, const BatchDesc &b, int64_t row)
{
    RowIn in;
    in.k = ReadKey(p.key, b, row, kKind);
    in.nulls = 0;
#pragma unroll
    for (int i = 0; i < kRegInputs; ++i) {
        in.v[i] = 0;
        if (i < p.nRegInputs) {
            const int c = p.regInput[i];
            in.v[i] = LoadBitsRO(b.cols[c], row, p.regWidth[i]);
            in.nulls |= (NullRO(b.nulls[c], row) ? 1u : 0u) << i;
        }
    }
    return in;
}

__device__ __forceinline__ uint64_t CachedBits(const AccSpec &s, const RowIn &in)
{
    uint64_t r = 0;
#pragma unroll
    for (int i = 0; i < kRegInputs; ++i) {
        r = (i == s.reg) ? in.v[i] : r;
    }
    return r;
}

__device__ __forceinline__ int64_t AccInt(const AccSpec &s, const BatchDesc &b, int64_t row, const RowIn &in)
{
    return s.reg >= 0 ? SignExtend(CachedBits(s, in), s.inWidth) : LoadInt(b.cols[s.input], row, s.inWidth);
}

__device__ __forceinline__ double AccDouble(const AccSpec &s, const BatchDesc &b, int64_t row, const RowIn &in)
{
    if (s.reg < 0) {
        return LoadAsDouble(b.cols[s.input], row, s.inKind, s.inWidth);
    }
    const uint64_t bits = CachedBits(s, in);
    if (s.inKind == IN_DOUBLE) {
        return __longlong_as_double(static_cast<long long>(bits));
    }
    if (s.inKind == IN_FLOAT) {
        return static_cast<double>(__int_as_float(static_cast<int>(bits)));
    }
    return static_cast<double>(SignExtend(bits, s.inWidth));
}

__device__ __forceinline__ bool AccNull(const AccSpec &s, const BatchDesc &b, int64_t row, const RowIn &in)
{
    return s.reg >= 0 ? ((in.nulls >> s.reg) & 1u) != 0 : RowIsNull(b.nulls[s.input], row);
}

__device__ __forceinline__ void Red(uint64_t *w, uint64_t v)
{
    if (v != 0) {
        atomicAdd(reinterpret_cast<unsigned long long *>(w), static_cast<unsigned long long>(v));
    }
}

// ------------------------------------------------------------------ VARCHAR min / max
// Order of the strings of dictionary ids a and b of input `input`: bytes compared as unsigned,
// a proper prefix first (std::string_view::compare, as the reference's MIN/MAX of VARCHAR).
__device__ __forceinline__ int CompareDictStrings(const AggLaunch &p, int input, int64_t a, int64_t b)
{
    const int64_t *off = p.strOff[input];
    const uint8_t *chars = p.strChars[input];
    const int64_t la = off[a + 1] - off[a];
    const int64_t lb = off[b + 1] - off[b];
    const uint8_t *x = chars + off[a];
    const uint8_t *y = chars + off[b];
    const int64_t n = la < lb ? la : lb;
    for (int64_t i = 0; i < n; ++i) {
        if (x[i] != y[i]) {
            return x[i] < y[i] ? -1 : 1;
        }
    }
    return la < lb ? -1 : (la > lb ? 1 : 0);
}

// Lock-free min / max of dictionary ids by their strings: a CAS succeeds only with a strictly
// better string, so every retry follows another thread's improvement and the loop ends.
__device__ __forceinline__ void AtomicStrMinMax(const AggLaunch &p, int input, uint64_t *w, int64_t id, bool isMin)
{
    unsigned long long *a = reinterpret_cast<unsigned long long *>(w);
    unsigned long long cur = *reinterpret_cast<volatile unsigned long long *>(a);
    while (true) {
        if (static_cast<int64_t>(cur) >= 0) {
            if (static_cast<int64_t>(cur) == id) {
                return;
            }
            const int c = CompareDictStrings(p, input, id, static_cast<int64_t>(cur));
            if (isMin ? c >= 0 : c <= 0) {
                return;
            }
        }
        const unsigned long long prev = atomicCAS(a, cur, static_cast<unsigned long long>(id));
        if (prev == cur) {
            return;
        }
        cur = prev;
    }
}

// Double sums that are added to row by row: the first kPlainSumRows rows of a slot of the global table,
// of a shared table in front of it or of a partition's shared table (by their COUNT_ALL arrival order)
// are added with a plain atomic add, the later ones with the compensated add.  Such a slot
// therefore leaves at most kPlainSumRows additions
// uncompensated, whose rounding errors add up to at most kPlainSumRows * 2^-53 * sum|x| (the
// slots of one group hold disjoint rows, so the bound holds for the group too): 7.1e-15 of
// sum|x| for 64.  Shared-table partials are merged compensated.  (2048 plain rows, 2.3e-13,
// measured no faster on the uniform workload: 190.7 us against 182-192 us.)  The states per thread, the
// steps (small calls, radix passes) and the batched tasks' units compensate every addition.
constexpr unsigned long long kPlainSumRows = 64;

__device__ __forceinline__ void AddDoubleState(uint64_t *w, double x, unsigned long long arrival)
{
    if (arrival < kPlainSumRows) {
        atomicAdd(reinterpret_cast<double *>(w), x);  // result unused: a fire-and-forget add
    } else {
        AtomicAddCompensated(w, x, 0.0);
    }
}

// ------------------------------------------------------------------ decimal128 min / max
// The state is a 16-byte (low, high) word pair; its initial value is +-(10^38 - 1), the
// reference's GetMax<Decimal128> (min_aggregator.h:31-34).
constexpr uint64_t kDec38MaxLo = 687399551400673279ull;
constexpr uint64_t kDec38MaxHi = 5421010862427522170ull;
constexpr uint64_t kDec38MinLo = ~kDec38MaxLo + 1ull;  // two's complement of 10^38 - 1
constexpr uint64_t kDec38MinHi = ~kDec38MaxHi;          // the low word is not zero: no carry

struct alignas(16) Dec128Word {
    unsigned long long lo;
    unsigned long long hi;
};

__device__ __forceinline__ void InitMinMax128(int kind, uint64_t *w)
{
    w[0] = kind == ACC_XMIN ? kDec38MaxLo : kDec38MinLo;
    w[1] = kind == ACC_XMIN ? kDec38MaxHi : kDec38MinHi;
}

__device__ __forceinline__ bool IsInitMinMax128(int kind, const uint64_t *w)
{
    return kind == ACC_XMIN ? (w[0] == kDec38MaxLo && w[1] == kDec38MaxHi) : (w[0] == kDec38MinLo && w[1] == kDec38MinHi);
}

// Lock-free 128-bit min / max: the current value is read with a no-op compare-and-swap (one
// atomic 16-byte read), and a CAS installs the value only while it is strictly better, so every
// retry follows another thread's improvement and the loop ends.
__device__ __forceinline__ void AtomicMinMax128(uint64_t *w, uint64_t lo, uint64_t hi, bool isMin)
{
    Dec128Word *a = reinterpret_cast<Dec128Word *>(w);
    Dec128Word val;
    val.lo = lo;
    val.hi = hi;
    Dec128Word cur = atomicCAS(a, val, val);
    while (true) {
        const int64_t vh = static_cast<int64_t>(hi);
        const int64_t ch = static_cast<int64_t>(cur.hi);
        const bool less = vh < ch || (vh == ch && lo < cur.lo);
        const bool greater = vh > ch || (vh == ch && lo > cur.lo);
        if (isMin ? !less : !greater) {
            return;
        }
        const Dec128Word prev = atomicCAS(a, cur, val);
        if (prev.lo == cur.lo && prev.hi == cur.hi) {
            return;
        }
        cur = prev;
    }
}

// ------------------------------------------------------------------ state updates
// `st` points at the group's state words, in shared or global memory.
__device__ __forceinline__ void UpdateStates(const AggLaunch &p, const BatchDesc &b, int64_t row, const RowIn &in,
    uint64_t *st)
{
    unsigned long long arrival = kPlainSumRows;  // rows of the slot before this one (COUNT_ALL is accs[0])
    for (int a = 0; a < p.nAccs; ++a) {
        const AccSpec &s = p.accs[a];
        uint64_t *w = st + s.word;
        if (s.kind == ACC_COUNT_ALL) {
            arrival = atomicAdd(reinterpret_cast<unsigned long long *>(w), 1ull);
            continue;
        }
        const bool isNull = AccNull(s, b, row, in);
        if (s.kind == ACC_NULLS) {
            if (isNull) {
                atomicAdd(reinterpret_cast<unsigned long long *>(w), 1ull);
            }
            continue;
        }
        if (isNull) {
            continue;
        }
        switch (s.kind) {
            case ACC_ISUM:
                Red(w, static_cast<uint64_t>(AccInt(s, b, row, in)));
                break;
            case ACC_WSUM2: {
                const int64_t x = AccInt(s, b, row, in);
                const uint64_t m = x >= 0 ? static_cast<uint64_t>(x) : 0ull - static_cast<uint64_t>(x);
                uint64_t *side = x >= 0 ? w : w + 2;
                Red(side, m & 0xffffffffull);
                Red(side + 1, m >> 32);
                break;
            }
            case ACC_WSUM3: {
                const uint64_t *v = static_cast<const uint64_t *>(b.cols[s.input]) + 2 * row;
                uint64_t lo = v[0];
                uint64_t hi = v[1];
                uint64_t *side = w;
                if (static_cast<int64_t>(hi) < 0) {  // magnitude = -(hi:lo)
                    lo = ~lo + 1;
                    hi = ~hi + (lo == 0 ? 1u : 0u);
                    side = w + 4;
                }
                Red(side, lo & 0xffffffffull);
                Red(side + 1, lo >> 32);
                Red(side + 2, hi & 0xffffffffull);
                Red(side + 3, hi >> 32);
                break;
            }
            case ACC_DSUM:
                AddDoubleState(w, AccDouble(s, b, row, in), arrival);
                break;
            case ACC_IMIN:
                AtomicMinI64(w, AccInt(s, b, row, in));
                break;
            case ACC_IMAX:
                AtomicMaxI64(w, AccInt(s, b, row, in));
                break;
            case ACC_DMIN: {
                const double x = AccDouble(s, b, row, in);
                if (!isnan(x)) {
                    AtomicMinI64(w, OrderedFromDouble(x));
                }
                break;
            }
            case ACC_DMAX: {
                const double x = AccDouble(s, b, row, in);
                if (!isnan(x)) {
                    AtomicMaxI64(w, OrderedFromDouble(x));
                }
                break;
            }
            case ACC_SMIN:
            case ACC_SMAX:
                AtomicStrMinMax(p, s.input, w, AccInt(s, b, row, in), s.kind == ACC_SMIN);
                break;
            case ACC_XMIN:
            case ACC_XMAX: {
                const uint64_t *v = static_cast<const uint64_t *>(b.cols[s.input]) + 2 * row;
                AtomicMinMax128(w, v[0], v[1], s.kind == ACC_XMIN);
                break;
            }
            default:
                break;
        }
    }
}

// Merge a partial state (shared table entry or spilled record) into `dst`.
__device__ __forceinline__ void MergeStates(const AggLaunch &p, const AccSpec *accs, int nAccs, const uint64_t *src,
    uint64_t *dst)
{
    for (int a = 0; a < nAccs; ++a) {
        const AccSpec &s = accs[a];
        const uint64_t *v = src + s.word;
        uint64_t *w = dst + s.word;
        switch (s.kind) {
            case ACC_COUNT_ALL:
            case ACC_NULLS:
            case ACC_ISUM:
                if (v[0] != 0) {
                    atomicAdd(reinterpret_cast<unsigned long long *>(w), static_cast<unsigned long long>(v[0]));
                }
                break;
            case ACC_WSUM2:
            case ACC_WSUM3:
                // chunk sums add word by word
                for (int j = 0; j < (s.kind == ACC_WSUM2 ? 4 : 8); ++j) {
                    Red(w + j, v[j]);
                }
                break;
            case ACC_DSUM: {
                double s0 = __longlong_as_double(static_cast<long long>(v[0]));
                double c0 = __longlong_as_double(static_cast<long long>(v[1]));
                if (s0 != 0.0 || c0 != 0.0) {
                    AtomicAddCompensated(w, s0, c0);
                }
                break;
            }
            case ACC_IMIN:
            case ACC_DMIN:
                if (static_cast<int64_t>(v[0]) != s.init) {
                    AtomicMinI64(w, static_cast<int64_t>(v[0]));
                }
                break;
            case ACC_IMAX:
            case ACC_DMAX:
                if (static_cast<int64_t>(v[0]) != s.init) {
                    AtomicMaxI64(w, static_cast<int64_t>(v[0]));
                }
                break;
            case ACC_SMIN:
            case ACC_SMAX:
                if (static_cast<int64_t>(v[0]) >= 0) {
                    AtomicStrMinMax(p, s.input, w, static_cast<int64_t>(v[0]), s.kind == ACC_SMIN);
                }
                break;
            case ACC_XMIN:
            case ACC_XMAX:
                if (!IsInitMinMax128(s.kind, v)) {
                    AtomicMinMax128(w, v[0], v[1], s.kind == ACC_XMIN);
                }
                break;
            default:
                break;
        }
    }
}

__device__ __forceinline__ void InitStates(const AccSpec *accs, int nAccs, int stateWords, uint64_t *st)
{
    for (int i = 0; i < stateWords; ++i) {
        st[i] = 0;
    }
    for (int a = 0; a < nAccs; ++a) {
        st[accs[a].word] = static_cast<uint64_t>(accs[a].init);
        if (accs[a].kind == ACC_XMIN || accs[a].kind == ACC_XMAX) {
            InitMinMax128(accs[a].kind, st + accs[a].word);
        }
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

// ------------------------------------------------------------------ global table
// Returns the slot index or -1 when no slot was found within maxProbe probes.
__device__ __forceinline__ int64_t GlobalFind(const AggTable &t, const KeySpec &ks, const RowKey &k, int maxProbe,
    int32_t *error, bool *inserted, long long waitBudget, int kind)
{
    *inserted = false;
    if (k.special >= 0) {
        const uint64_t slot = t.capacity + static_cast<uint64_t>(k.special);
        if (t.specialUsed[k.special] == 0) {
            atomicExch(&t.specialUsed[k.special], 1u);
        }
        return static_cast<int64_t>(slot);
    }
    const uint64_t mask = t.capacity - 1;
    uint64_t i = k.hash & mask;
    if (kind == KEY_SINGLE) {
        for (int probe = 0; probe < maxProbe; ++probe) {
            unsigned long long *kp = reinterpret_cast<unsigned long long *>(t.slots + i * t.slotWords);
            unsigned long long cur = *reinterpret_cast<volatile unsigned long long *>(kp);
            if (cur == k.w[0]) {
                return static_cast<int64_t>(i);
            }
            if (cur == kEmptyKey) {
                unsigned long long prev = atomicCAS(kp, kEmptyKey, k.w[0]);
                if (prev == kEmptyKey) {
                    *inserted = true;
                    return static_cast<int64_t>(i);
                }
                if (prev == k.w[0]) {
                    return static_cast<int64_t>(i);
                }
            }
            i = (i + 1) & mask;
        }
        return -1;
    }
    const uint64_t tag = PublishedTag(k.hash);
    for (int probe = 0; probe < maxProbe; ++probe) {
        uint64_t *slot = t.slots + i * t.slotWords;
        uint64_t cur = LoadAcquire(slot);
        if (cur == 0) {
            unsigned long long prev =
                atomicCAS(reinterpret_cast<unsigned long long *>(slot), 0ull, static_cast<unsigned long long>(kTagLocked));
            if (prev == 0) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    if (j < ks.words) {
                        slot[1 + j] = k.w[j];
                    }
                }
                StoreRelease(slot, tag);
                *inserted = true;
                return static_cast<int64_t>(i);
            }
            cur = prev;
        }
        if (cur == kTagLocked) {
            // Another thread is publishing this slot's key: wait a bounded time.
            long long start = clock64();
            while ((cur = LoadAcquire(slot)) == kTagLocked) {
                if (clock64() - start > waitBudget) {
                    SetError(error, 7);
                    return -1;
                }
            }
        }
        if (cur == tag) {
            bool eq = true;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                eq = eq && (j >= ks.words || slot[1 + j] == k.w[j]);
            }
            if (eq) {
                return static_cast<int64_t>(i);
            }
        }
        i = (i + 1) & mask;
    }
    return -1;
}

// ------------------------------------------------------------------ shared-memory table
// Same layout as the global table (slotWords words per slot), nSlots slots, no special
// slots (those rows go straight to the global table).  Returns the slot or -1.
__device__ __forceinline__ int SmemFind(uint64_t *sm, int nSlots, int slotWords, const KeySpec &ks, const RowKey &k,
    int kind, int maxProbe = kSmemProbe)
{
    int i = static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(k.hash >> 32)) * nSlots) >> 32);
    if (kind == KEY_SINGLE) {
        for (int probe = 0; probe < maxProbe; ++probe) {
            unsigned long long *kp = reinterpret_cast<unsigned long long *>(sm + static_cast<int64_t>(i) * slotWords);
            unsigned long long cur = *reinterpret_cast<volatile unsigned long long *>(kp);
            if (cur == k.w[0]) {
                return i;
            }
            if (cur == kEmptyKey) {
                unsigned long long prev = atomicCAS(kp, kEmptyKey, k.w[0]);
                if (prev == kEmptyKey || prev == k.w[0]) {
                    return i;
                }
            }
            if (++i == nSlots) {
                i = 0;
            }
        }
        return -1;
    }
    const uint64_t tag = PublishedTag(k.hash);
    for (int probe = 0; probe < maxProbe; ++probe) {
        uint64_t *slot = sm + static_cast<int64_t>(i) * slotWords;
        volatile uint64_t *vs = slot;
        uint64_t cur = vs[0];
        if (cur == 0) {
            unsigned long long prev =
                atomicCAS(reinterpret_cast<unsigned long long *>(slot), 0ull, static_cast<unsigned long long>(kTagLocked));
            if (prev == 0) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    if (j < ks.words) {
                        vs[1 + j] = k.w[j];
                    }
                }
                __threadfence_block();
                vs[0] = tag;
                return i;
            }
            cur = prev;
        }
        if (cur == kTagLocked) {
            int spins = 0;
            while ((cur = vs[0]) == kTagLocked) {
                if (++spins > (1 << 20)) {
                    return -1;  // give up on the shared table; the row goes global
                }
            }
        }
        if (cur == tag) {
            __threadfence_block();
            bool eq = true;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                eq = eq && (j >= ks.words || vs[1 + j] == k.w[j]);
            }
            if (eq) {
                return i;
            }
        }
        if (++i == nSlots) {
            i = 0;
        }
    }
    return -1;
}

__device__ __forceinline__ bool SlotOccupied(const KeySpec &ks, uint64_t firstWord)
{
    return ks.kind == KEY_SINGLE ? firstWord != kEmptyKey : (firstWord != 0 && firstWord != kTagLocked);
}

__device__ __forceinline__ void QueueRetry(const AggLaunch &p, int32_t batch, int64_t row)
{
    unsigned int pos = atomicAdd(p.nRetry, 1u);
    if (pos < p.retryCap) {
        p.retry[pos] = (static_cast<unsigned long long>(batch) << 32) | static_cast<unsigned long long>(row);
    } else {
        SetError(p.error, 4);  // queue overflow: the host sized it for every row, so this is a bug
    }
}

template <int kKind>
__device__ __forceinline__ void ProcessRow(const AggLaunch &p, int32_t batchIdx, const BatchDesc &b, int64_t row,
    const RowIn &in, uint64_t *sm, int smSlots, unsigned int *newGroups)
{
    const int sw = p.table.slotWords;
    const int kw = p.table.keyWords;
    if (smSlots > 0 && in.k.special < 0) {
        int i = SmemFind(sm, smSlots, p.smemStride, p.key, in.k, kKind);
        if (i >= 0) {
            UpdateStates(p, b, row, in, sm + static_cast<int64_t>(i) * p.smemStride + kw);
            return;
        }
    }
    bool inserted = false;
    int64_t g = GlobalFind(p.table, p.key, in.k, p.maxProbe, p.error, &inserted, p.waitBudget, kKind);
    if (g < 0) {
        QueueRetry(p, batchIdx, row);
        return;
    }
    if (inserted) {
        atomicAdd(newGroups, 1u);
    }
    UpdateStates(p, b, row, in, p.table.slots + g * sw + kw);
}

// Spill records: [key words (keyWords)][state words], slotWords words each.
struct SpillArgs {
    uint64_t *spill;
    unsigned int *nSpill;
    uint32_t spillCap;
    const uint64_t *spillIn;
    uint32_t nSpillIn;
};

// The key of a record or a slot.
template <int kKind> __device__ __forceinline__ RowKey RecordKey(const AggLaunch &p, const uint64_t *rec)
{
    RowKey k;
    k.special = -1;
    k.w[0] = k.w[1] = k.w[2] = 0;
    if (kKind == KEY_SINGLE) {
        k.w[0] = rec[0];
        k.hash = Mix64(k.w[0]);
    } else {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            k.w[j] = j < p.key.words ? rec[1 + j] : 0ull;
        }
        k.hash = KeyWordsHash(k, p.key.words);
    }
    return k;
}

template <int kKind>
__device__ __forceinline__ void MergeRecord(const AggLaunch &p, const SpillArgs &sp, const uint64_t *rec,
    unsigned int *newGroups)
{
    const int sw = p.table.slotWords;
    const int kw = p.table.keyWords;
    const RowKey k = RecordKey<kKind>(p, rec);
    bool inserted = false;
    int64_t g = GlobalFind(p.table, p.key, k, p.maxProbe, p.error, &inserted, p.waitBudget, kKind);
    if (g < 0) {
        unsigned int pos = atomicAdd(sp.nSpill, 1u);
        if (pos < sp.spillCap) {
            uint64_t *dst = sp.spill + static_cast<int64_t>(pos) * sw;
            for (int i = 0; i < sw; ++i) {
                dst[i] = rec[i];
            }
        } else {
            SetError(p.error, 4);
        }
        return;
    }
    if (inserted) {
        atomicAdd(newGroups, 1u);
    }
    MergeStates(p, p.accs, p.nAccs, rec + kw, p.table.slots + g * sw + kw);
}

// ------------------------------------------------------------------ dense shared tables
// Slots without free ones between them (0 and 1: the NULL and the EMPTY key), found through an index of
// 32-bit words, a 16-bit tag and a slot number, that is at most half full.
constexpr int kSpecialSlots = 2;
constexpr unsigned int kIndexLocked = 0xffffffffu;
constexpr unsigned int kIndexFull = 0xfffffffeu;

// The slot of key k among the groups (kSpecialSlots and up), taking a new one if need be, or -1: the
// table is full (a key that once misses then misses every time: the entry it would take stays full).
__device__ __forceinline__ int FindGroup(uint64_t *sm, unsigned int *index, unsigned int indexMask, unsigned int *used,
    unsigned int nSlots, int sw, const KeySpec &ks, const RowKey &k, int kind)
{
    const unsigned int tag = static_cast<unsigned int>(k.hash >> 48) << 16;
    unsigned int i = static_cast<unsigned int>(k.hash >> 32) & indexMask;
    for (unsigned int probe = 0; probe <= indexMask; ++probe) {
        volatile unsigned int *ve = index + i;
        unsigned int e = *ve;
        if (e == 0) {
            e = atomicCAS(index + i, 0u, kIndexLocked);
            if (e == 0) {
                const unsigned int slot = atomicAdd(used, 1u);
                if (slot >= nSlots) {
                    *ve = kIndexFull;
                    return -1;
                }
                volatile uint64_t *to = sm + static_cast<int64_t>(slot + kSpecialSlots) * sw;
                if (kind == KEY_SINGLE) {
                    to[0] = k.w[0];
                } else {
                    to[0] = PublishedTag(k.hash);
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        if (j < ks.words) {
                            to[1 + j] = k.w[j];
                        }
                    }
                }
                __threadfence_block();
                *ve = tag | (slot + kSpecialSlots);
                return static_cast<int>(slot + kSpecialSlots);
            }
        }
        if (e == kIndexLocked) {
            // Another thread is writing this entry's key: a handful of instructions, then it publishes.
            int spins = 0;
            while ((e = *ve) == kIndexLocked) {
                if (++spins > (1 << 20)) {
                    return -2;
                }
            }
        }
        if (e == kIndexFull) {
            return -1;
        }
        if ((e & 0xffff0000u) == tag) {
            __threadfence_block();
            const int slot = static_cast<int>(e & 0xffffu);
            const volatile uint64_t *at = sm + static_cast<int64_t>(slot) * sw;
            bool eq;
            if (kind == KEY_SINGLE) {
                eq = at[0] == k.w[0];
            } else {
                eq = true;
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    eq = eq && (j >= ks.words || at[1 + j] == k.w[j]);
                }
            }
            if (eq) {
                return slot;
            }
        }
        i = (i + 1) & indexMask;
    }
    return -1;
}

__device__ __forceinline__ void InitSlot(const AggLaunch &p, uint64_t *slot)
{
    slot[0] = (p.key.kind == KEY_SINGLE) ? kEmptyKey : 0ull;
    for (int j = 1; j < p.table.keyWords; ++j) {
        slot[j] = 0;
    }
    InitStates(p.accs, p.nAccs, p.stateWords, slot + p.table.keyWords);
}

__device__ __forceinline__ double AsDouble(uint64_t bits, int inKind, int width)
{
    if (inKind == IN_DOUBLE) {
        return __longlong_as_double(static_cast<long long>(bits));
    }
    if (inKind == IN_FLOAT) {
        return static_cast<double>(__int_as_float(static_cast<int>(bits)));
    }
    return static_cast<double>(SignExtend(bits, width));
}

}  // namespace
}  // namespace omg
