// Group-by with a handful of groups.
//
// With few groups the shared tables' atomics are all on the same words: 2^22 rows of 6 groups, two INT keys
// and six aggregates ran 1.22 ms, and 0.18 ms here (507 instructions a warp's row, a third of them the packed
// key, at 0.33 of the issue slots and 0.39 of the FP64 pipe; 0.144 ms and 480 without the errors of the double
// sums, three FP64 operations a row; their chains side by side for a step's rows measured no faster).  Here every thread keeps states of its own for every group, in planes of shared
// memory where the threads of a warp are side by side: no atomics and no bank conflicts.  A sum of doubles has a
// plane for the rounding errors of its additions.  Exact sums move to the CTA's state of the group every 64
// rows (magnitudes of up to 64 values below 2^57), and at the end a warp adds up each group's private states
// and the CTA's records are merged into the global table.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "agg_device.cuh"
#include "agg_few.h"
#include "device_common.cuh"
#include "launch.h"

namespace omg {
namespace {

constexpr int kFewRows = 4;  // rows per thread per step: their loads are in flight together
constexpr size_t kFewSmemBytes = 110 * 1024;  // two CTAs per SM
constexpr unsigned int kFoldRows = 64;
constexpr int kFewIndex = 256;

template <class T, int kThreads> __device__ __forceinline__ T *Plane(unsigned char *smem, int off, int group)
{
    return reinterpret_cast<T *>(smem + off) + group * kThreads + threadIdx.x;
}

__device__ __forceinline__ void AddTwoSum(double &s, double &c, double x)
{
    const double sum = __dadd_rn(s, x);
    if (isfinite(sum)) {
        c = __dadd_rn(c, SumError(s, x, sum));
    }
    s = sum;
}

// An input's values (up to 8 bytes; width 0: none) and NULL bits of the thread's rows.
struct FewInput {
    uint64_t bits[kFewRows];
    uint32_t null;
};

template <int kThreads>
__device__ __forceinline__ void LoadFew(const BatchRows<kThreads> &rows, int input, int width, uint32_t live,
    FewInput &in)
{
    in.null = 0;
    if (input < 0) {
        return;
    }
    if (width > 0) {
        LoadBitsRows<kFewRows>([&](int k) { return rows.At(input, width, k); }, width, live, in.bits);
    }
    if (rows.Nullable(input)) {
        in.null = rows.Nulls<kFewRows>(input, live);
    }
}

// Accumulator a over the thread's rows (bit k of live); at[k]: the element of row k's group in a plane;
// fold: bit k: the thread's 64th row of its group, or 128th and so on; states[k]: the CTA's states of it.
__device__ __forceinline__ void ApplyFew(const AggLaunch &p, const FewLayout &l, int a, const FewInput &in, uint32_t live,
    const int (&at)[kFewRows], uint32_t fold, uint64_t *const (&states)[kFewRows], unsigned char *smem)
{
    const AccSpec &s = p.accs[a];
    unsigned char *plane = smem + l.off[a];
    uint32_t has = live & ~in.null;
    switch (s.kind) {
        case ACC_NULLS:
#pragma unroll
            for (int k = 0; k < kFewRows; ++k) {
                if (((live & in.null) >> k) & 1u) {
                    ++reinterpret_cast<unsigned int *>(plane)[at[k]];
                }
            }
            break;
        case ACC_ISUM:
#pragma unroll
            for (int k = 0; k < kFewRows; ++k) {
                if ((has >> k) & 1u) {
                    reinterpret_cast<uint64_t *>(plane)[at[k]] += static_cast<uint64_t>(SignExtend(in.bits[k], s.inWidth));
                }
            }
            break;
        case ACC_WSUM2: {
            uint64_t *pos = reinterpret_cast<uint64_t *>(plane);
            uint64_t *neg = reinterpret_cast<uint64_t *>(plane + l.planeStep[a]);
#pragma unroll
            for (int k = 0; k < kFewRows; ++k) {
                uint64_t *to = states[k] + s.word;
                if ((has >> k) & 1u) {
                    const int64_t x = SignExtend(in.bits[k], s.inWidth);
                    const uint64_t m = x >= 0 ? static_cast<uint64_t>(x) : 0ull - static_cast<uint64_t>(x);
                    if ((m >> 57) != 0) {
                        SharedAdd(to + (x >= 0 ? 0 : 2), m & 0xffffffffull);
                        SharedAdd(to + (x >= 0 ? 1 : 3), m >> 32);
                    } else {
                        (x >= 0 ? pos : neg)[at[k]] += m;
                    }
                }
                if ((fold >> k) & 1u) {
                    const uint64_t u = pos[at[k]];
                    const uint64_t v = neg[at[k]];
                    SharedAdd(to, u & 0xffffffffull);
                    SharedAdd(to + 1, u >> 32);
                    SharedAdd(to + 2, v & 0xffffffffull);
                    SharedAdd(to + 3, v >> 32);
                    pos[at[k]] = 0;
                    neg[at[k]] = 0;
                }
            }
            break;
        }
        case ACC_DSUM: {
            double *sum = reinterpret_cast<double *>(plane);
            double *err = reinterpret_cast<double *>(plane + l.planeStep[a]);
#pragma unroll
            for (int k = 0; k < kFewRows; ++k) {
                if ((has >> k) & 1u) {
                    // Once a sum is not finite it stays so, and its errors (NaN then) are not looked at.
                    const double x = AsDouble(in.bits[k], s.inKind, s.inWidth);
                    const double old = sum[at[k]];
                    const double next = __dadd_rn(old, x);
                    sum[at[k]] = next;
                    err[at[k]] = __dadd_rn(err[at[k]], SumError(old, x, next));
                }
            }
            break;
        }
        case ACC_DMIN:
        case ACC_DMAX:
        case ACC_IMIN:
        case ACC_IMAX: {
            long long x[kFewRows];
            if (s.kind == ACC_IMIN || s.kind == ACC_IMAX) {
#pragma unroll
                for (int k = 0; k < kFewRows; ++k) {
                    x[k] = SignExtend(in.bits[k], s.inWidth);
                }
            } else {
#pragma unroll
                for (int k = 0; k < kFewRows; ++k) {
                    const double d = AsDouble(in.bits[k], s.inKind, s.inWidth);
                    has &= ~((isnan(d) ? 1u : 0u) << k);
                    x[k] = OrderedFromDouble(d);
                }
            }
            long long *w = reinterpret_cast<long long *>(plane);
            if (s.kind == ACC_IMIN || s.kind == ACC_DMIN) {
#pragma unroll
                for (int k = 0; k < kFewRows; ++k) {
                    if (((has >> k) & 1u) != 0) {
                        w[at[k]] = min(w[at[k]], x[k]);
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < kFewRows; ++k) {
                    if (((has >> k) & 1u) != 0) {
                        w[at[k]] = max(w[at[k]], x[k]);
                    }
                }
            }
            break;
        }
        default:
            break;
    }
}

// Add up the private states of group `group` (by one warp) into the CTA's slot.
template <int kThreads>
__device__ __forceinline__ void FoldGroup(const AggLaunch &p, const FewLayout &l, unsigned char *smem, int group,
    uint64_t *state)
{
    const int lane = threadIdx.x & 31;
    for (int a = 0; a < p.nAccs; ++a) {
        const AccSpec &s = p.accs[a];
        const int off = l.off[a];
        if (off < 0) {
            continue;
        }
        uint64_t *w = state + s.word;
        const unsigned int *n32 = reinterpret_cast<const unsigned int *>(smem + off) + group * kThreads;
        const uint64_t *n64 = reinterpret_cast<const uint64_t *>(smem + off) + group * kThreads;
        if (s.kind == ACC_DSUM) {
            const uint64_t *e64 = n64 + l.planeStep[a] / 8;
            double sum = 0.0, err = 0.0;
            for (int t = lane; t < kThreads; t += 32) {
                AddTwoSum(sum, err, __longlong_as_double(static_cast<long long>(n64[t])));
                err = __dadd_rn(err, __longlong_as_double(static_cast<long long>(e64[t])));
            }
            for (int o = 16; o > 0; o >>= 1) {
                const double os = __shfl_xor_sync(0xffffffffu, sum, o);
                const double oe = __shfl_xor_sync(0xffffffffu, err, o);
                AddTwoSum(sum, err, os);
                err = __dadd_rn(err, oe);
            }
            if (lane == 0) {
                double s0 = __longlong_as_double(static_cast<long long>(w[0]));
                double c0 = __longlong_as_double(static_cast<long long>(w[1]));
                AddTwoSum(s0, c0, sum);
                w[0] = static_cast<uint64_t>(__double_as_longlong(s0));
                w[1] = static_cast<uint64_t>(__double_as_longlong(__dadd_rn(c0, err)));
            }
            continue;
        }
        if (s.kind == ACC_IMIN || s.kind == ACC_IMAX || s.kind == ACC_DMIN || s.kind == ACC_DMAX) {
            const bool isMin = s.kind == ACC_IMIN || s.kind == ACC_DMIN;
            long long x = static_cast<long long>(s.init);
            for (int t = lane; t < kThreads; t += 32) {
                const long long v = static_cast<long long>(n64[t]);
                x = isMin ? min(x, v) : max(x, v);
            }
            for (int o = 16; o > 0; o >>= 1) {
                const long long v = __shfl_xor_sync(0xffffffffu, x, o);
                x = isMin ? min(x, v) : max(x, v);
            }
            if (lane == 0) {
                w[0] = static_cast<uint64_t>(x);
            }
            continue;
        }
        const int planes = s.kind == ACC_WSUM2 ? 2 : 1;
        for (int side = 0; side < planes; ++side) {
            const uint64_t *n = n64 + side * (l.planeStep[a] / 8);
            unsigned long long lo = 0, hi = 0;  // chunk sums of the magnitudes, or the plain sum in lo
            for (int t = lane; t < kThreads; t += 32) {
                if (s.kind == ACC_WSUM2) {
                    lo += n[t] & 0xffffffffull;
                    hi += n[t] >> 32;
                } else {
                    lo += s.kind == ACC_ISUM ? n64[t] : n32[t];
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                lo += __shfl_xor_sync(0xffffffffu, lo, o);
                hi += __shfl_xor_sync(0xffffffffu, hi, o);
            }
            if (lane == 0) {
                w[2 * side] += lo;
                if (s.kind == ACC_WSUM2) {
                    w[2 * side + 1] += hi;
                }
            }
        }
    }
}

template <int kKind, int kThreads>
__global__ void __launch_bounds__(kThreads, 2) AggFewKernel(const __grid_constant__ AggLaunch p,
    const __grid_constant__ FewLayout l, const __grid_constant__ SpillArgs sp)
{
    // The private planes (from byte 0), then the CTA's slots and their index.
    extern __shared__ __align__(16) unsigned char smem8[];
    __shared__ unsigned int index[kFewIndex];
    __shared__ unsigned int used;
    __shared__ unsigned int newGroups;
    const int sw = p.table.slotWords;
    const int kw = p.table.keyWords;
    const int nSlots = l.maxGroups + l.firstSlot - kSpecialSlots;  // beside the special ones
    const int nAll = nSlots + kSpecialSlots;
    uint64_t *slots = reinterpret_cast<uint64_t *>(smem8 + l.smemBytes) - static_cast<int64_t>(nAll) * sw;
    uint64_t *st = slots + l.firstSlot * sw + kw;
    for (int i = threadIdx.x; i < nAll; i += kThreads) {
        InitSlot(p, slots + static_cast<int64_t>(i) * sw);
    }
    for (int i = threadIdx.x; i < kFewIndex; i += kThreads) {
        index[i] = 0;
    }
    for (int a = 0; a < p.nAccs; ++a) {
        const AccSpec &s = p.accs[a];
        if (l.off[a] < 0) {
            continue;
        }
        for (int g = 0; g < l.maxGroups; ++g) {
            if (s.kind == ACC_COUNT_ALL || s.kind == ACC_NULLS) {
                *Plane<unsigned int, kThreads>(smem8, l.off[a], g) = 0;
            } else {
                *Plane<uint64_t, kThreads>(smem8, l.off[a], g) = s.kind == ACC_DSUM || s.kind == ACC_ISUM || s.kind == ACC_WSUM2
                    ? 0ull : static_cast<uint64_t>(s.init);
                if (s.kind == ACC_WSUM2 || s.kind == ACC_DSUM) {
                    *Plane<uint64_t, kThreads>(smem8, l.off[a] + l.planeStep[a], g) = 0;
                }
            }
        }
    }
    if (threadIdx.x == 0) {
        used = 0;
        newGroups = 0;
    }
    __syncthreads();
    for (int t = blockIdx.x; t < p.nTiles; t += gridDim.x) {
        const TileDesc tile = p.tiles[t];
        const BatchDesc &b = p.batches[tile.batch];
        for (int r0 = threadIdx.x; r0 < tile.rows; r0 += kFewRows * kThreads) {
            uint32_t live = 0;
#pragma unroll
            for (int k = 0; k < kFewRows; ++k) {
                live |= r0 + k * kThreads < tile.rows ? 1u << k : 0u;
            }
            const BatchRows<kThreads> rows{b, static_cast<int64_t>(tile.row0) + r0};
            // The first input's values come with the keys, each later one's with the work on the one before.
            FewInput in;
            LoadFew(rows, l.nInputs > 0 ? l.input[0] : -1, l.nInputs > 0 ? l.width[0] : 0, live, in);
            RowKey key[kFewRows];
            ReadKeys<kKind, kFewRows>(p.key, rows, live, key);
            int at[kFewRows];
            uint64_t *states[kFewRows];
            uint32_t fold = 0;
            uint32_t global = 0;  // rows whose group has no slot here
#pragma unroll
            for (int k = 0; k < kFewRows; ++k) {
                at[k] = 0;
                states[k] = st;
                if (((live >> k) & 1u) == 0) {
                    continue;
                }
                int slot;
                if (key[k].special >= 0) {
                    slot = key[k].special >= l.firstSlot ? key[k].special : -1;
                } else {
                    slot = FindGroup(slots, index, kFewIndex - 1, &used, nSlots, sw, p.key, key[k], kKind);
                    if (slot == -2) {
                        SetError(p.error, 7);
                    }
                }
                if (slot < 0) {
                    live &= ~(1u << k);
                    global |= slot == -1 ? 1u << k : 0u;
                    continue;
                }
                at[k] = (slot - l.firstSlot) * kThreads + threadIdx.x;
                states[k] = st + (slot - l.firstSlot) * sw;
                unsigned int *c = reinterpret_cast<unsigned int *>(smem8 + l.off[0]) + at[k];  // accs[0]: COUNT_ALL
                const unsigned int n = *c + 1;
                *c = n;
                fold |= n % kFoldRows == 0 ? 1u << k : 0u;
            }
            if (global != 0) {
#pragma unroll 1
                for (int k = 0; k < kFewRows; ++k) {
                    if ((global >> k) & 1u) {
                        const int64_t row = rows.row0 + k * kThreads;
                        ProcessRow<kKind>(p, tile.batch, b, row, LoadRow<kKind>(p, b, row), nullptr, 0, &newGroups);
                    }
                }
            }
            for (int i = 0; i < l.nInputs; ++i) {
                FewInput next;
                LoadFew(rows, i + 1 < l.nInputs ? l.input[i + 1] : -1, i + 1 < l.nInputs ? l.width[i + 1] : 0, live, next);
                for (int a = l.firstAcc[i]; a < l.firstAcc[i + 1]; ++a) {
                    ApplyFew(p, l, l.acc[a], in, live, at, fold, states, smem8);
                }
                in = next;
            }
        }
    }
    __syncthreads();
    const int nUsed = static_cast<int>(min(used, static_cast<unsigned int>(nSlots))) + kSpecialSlots;
    for (int slot = l.firstSlot + (threadIdx.x >> 5); slot < nUsed; slot += kThreads / 32) {
        FoldGroup<kThreads>(p, l, smem8, slot - l.firstSlot, slots + static_cast<int64_t>(slot) * sw + kw);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nUsed; i += kThreads) {
        uint64_t *slot = slots + static_cast<int64_t>(i) * sw;
        if (i >= kSpecialSlots) {
            MergeRecord<kKind>(p, sp, slot, &newGroups);
        } else if (slot[kw + p.accs[0].word] != 0) {
            atomicExch(&p.table.specialUsed[i], 1u);
            MergeStates(p, p.accs, p.nAccs, slot + kw, p.table.slots + (p.table.capacity + i) * sw + kw);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && newGroups != 0) {
        atomicAdd(p.table.groupCount, static_cast<unsigned long long>(newGroups));
    }
}

}  // namespace

bool LayoutAggFew(const AggLaunch &p, uint32_t nullable, uint64_t slots, FewLayout *l)
{
    int perGroup = 0;  // bytes of a thread's states of one group
    int errors = 0;    // of them, for the errors of double sums
    int bytes[kMaxAccs];
    bool keyNullable = false;
    for (int c = 0; c < p.key.nCols; ++c) {
        keyNullable = keyNullable || (p.key.kind == KEY_SINGLE && ((nullable >> p.key.cols[c].input) & 1u) != 0);
    }
    for (int a = 0; a < p.nAccs; ++a) {
        const AccSpec &s = p.accs[a];
        switch (s.kind) {
            case ACC_COUNT_ALL:
                bytes[a] = 4;
                break;
            case ACC_NULLS:
                bytes[a] = ((nullable >> s.input) & 1u) != 0 ? 4 : 0;
                break;
            case ACC_ISUM:
            case ACC_IMIN:
            case ACC_IMAX:
            case ACC_DMIN:
            case ACC_DMAX:
                bytes[a] = 8;
                break;
            case ACC_DSUM:
                errors += 8;
                bytes[a] = 16;
                break;
            case ACC_WSUM2:
                bytes[a] = 16;
                break;
            default:
                return false;
        }
        perGroup += bytes[a];
    }
    l->firstSlot = keyNullable ? 0 : kSpecialSlots;
    const int slotBytes = p.table.slotWords * 8;
    const int room = static_cast<int>(kFewSmemBytes) - kSpecialSlots * slotBytes - 16;
    auto fits = [&](int threads, int bytesPerGroup) {
        return std::min(room / (bytesPerGroup * threads + slotBytes), kFewIndex / 2);
    };
    // The line: as many groups as 256 threads have room for beside the errors of their double sums.  With the errors,
    // the most of them takes fewer threads: 2^24 rows, two-column key, 12 groups of six aggregates (192 threads) 0.86 ms
    // against 2.53 by the partitions' tables, 30 groups of one double sum (128 threads) 1.02 against 1.33; at 2^19
    // rows 0.16 against 0.24 and 0.20 against 0.16.
    const int most = fits(kFewMaxThreads, perGroup - errors);
    if (most - (kSpecialSlots - l->firstSlot) < 4 || slots > static_cast<uint64_t>(most + l->firstSlot)) {
        return false;
    }
    for (l->threads = kFewMaxThreads; l->threads > kFewMinThreads; l->threads -= 64) {
        if (slots <= static_cast<uint64_t>(fits(l->threads, perGroup) + l->firstSlot)) {
            break;
        }
    }
    l->maxGroups = fits(l->threads, perGroup);
    // 8-byte planes first, then the counters; the slots end the block on an 8-byte boundary.
    int at = 0;
    for (int pass = 0; pass < 2; ++pass) {
        for (int a = 0; a < p.nAccs; ++a) {
            const int unit = bytes[a] >= 8 ? 8 : 4;
            if (bytes[a] == 0) {
                l->off[a] = -1;
                l->planeStep[a] = 0;
            } else if ((pass == 0) == (unit == 8)) {
                l->off[a] = at;
                l->planeStep[a] = unit * l->threads * l->maxGroups;
                at += bytes[a] * l->threads * l->maxGroups;
            }
        }
    }
    // The accumulators by input.
    l->nInputs = 0;
    int n = 0;
    for (int i = 0; i < kMaxInputs; ++i) {
        const int first = n;
        int width = 0;
        for (int a = 1; a < p.nAccs; ++a) {
            if (p.accs[a].input == i && l->off[a] >= 0) {
                l->acc[n++] = static_cast<int16_t>(a);
                width = p.accs[a].kind != ACC_NULLS ? p.accs[a].inWidth : width;
            }
        }
        if (n > first) {
            l->input[l->nInputs] = static_cast<int16_t>(i);
            l->width[l->nInputs] = static_cast<int16_t>(width);
            l->firstAcc[l->nInputs++] = static_cast<int16_t>(first);
            l->firstAcc[l->nInputs] = static_cast<int16_t>(n);
        }
    }
    const int nAll = l->maxGroups + l->firstSlot;
    l->smemBytes = (at + nAll * slotBytes + 15) / 16 * 16;
    return true;
}

int LaunchAggFewGrid() { return DeviceSMCount() * 2; }

cudaError_t LaunchAggFew(const AggLaunch &p, const FewLayout &l, uint64_t *spill, unsigned int *nSpill,
    uint32_t spillCap, cudaStream_t stream)
{
    if (p.nTiles <= 0) {
        return cudaSuccess;
    }
    const SpillArgs sp{spill, nSpill, spillCap, nullptr, 0};
    const bool single = p.key.kind == KEY_SINGLE;
    auto kernel = l.threads == 256 ? (single ? AggFewKernel<KEY_SINGLE, 256> : AggFewKernel<KEY_PACKED, 256>)
        : l.threads == 192         ? (single ? AggFewKernel<KEY_SINGLE, 192> : AggFewKernel<KEY_PACKED, 192>)
                                   : (single ? AggFewKernel<KEY_SINGLE, 128> : AggFewKernel<KEY_PACKED, 128>);
    const cudaError_t err = EnsureDynamicSmem(reinterpret_cast<const void *>(kernel), kFewSmemBytes);
    if (err != cudaSuccess) {
        return err;
    }
    const int grid = p.nTiles < LaunchAggFewGrid() ? p.nTiles : LaunchAggFewGrid();
    kernel<<<grid, l.threads, l.smemBytes, stream>>>(p, l, sp);
    return cudaGetLastError();
}

}  // namespace omg
