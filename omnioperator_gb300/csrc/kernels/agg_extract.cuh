// Device functions that turn a group's states into its output row.
#pragma once

#include "agg_device.cuh"

namespace omg {
namespace {

// ------------------------------------------------------------------ output extraction
__device__ __forceinline__ void SetOutNull(uint8_t *nulls, uint64_t pos)
{
    atomicOr(reinterpret_cast<unsigned int *>(nulls) + (pos >> 5), 1u << (pos & 31));
}

__device__ __forceinline__ void StoreWidth(void *col, uint64_t pos, int width, uint64_t bits)
{
    switch (width) {
        case 1:
            static_cast<uint8_t *>(col)[pos] = static_cast<uint8_t>(bits);
            break;
        case 2:
            static_cast<uint16_t *>(col)[pos] = static_cast<uint16_t>(bits);
            break;
        case 4:
            static_cast<uint32_t *>(col)[pos] = static_cast<uint32_t>(bits);
            break;
        default:
            static_cast<uint64_t *>(col)[pos] = bits;
            break;
    }
}

// 10^38 - 1 as a 128-bit unsigned value (type/base_operations.h:20-21).
__device__ __forceinline__ unsigned __int128 Dec38Max()
{
    return (static_cast<unsigned __int128>(5421010862427522170ull) << 64) | 687399551400673279ull;
}

// Decode a WSUM accumulator: exact signed sum (as sign + 192-bit magnitude) and Sum|x|.
struct WideSum {
    bool negative;
    uint64_t mag[3];   // |sum|
    uint64_t abs[3];   // Sum|x| (saturated bit set in abs[2] top bit if it overflowed 192 bits)
};

__device__ __forceinline__ int Cmp192(const uint64_t *a, const uint64_t *b)
{
    for (int i = 2; i >= 0; --i) {
        if (a[i] != b[i]) {
            return a[i] < b[i] ? -1 : 1;
        }
    }
    return 0;
}

__device__ __forceinline__ void Sub192(const uint64_t *a, const uint64_t *b, uint64_t *r)
{
    uint64_t borrow = 0;
    for (int i = 0; i < 3; ++i) {
        uint64_t d = a[i] - b[i];
        uint64_t b1 = a[i] < b[i];
        uint64_t d2 = d - borrow;
        uint64_t b2 = d < borrow;
        r[i] = d2;
        borrow = b1 | b2;
    }
}

__device__ __forceinline__ void Add192(const uint64_t *a, const uint64_t *b, uint64_t *r)
{
    uint64_t carry = 0;
    for (int i = 0; i < 3; ++i) {
        uint64_t s = a[i] + b[i];
        uint64_t c1 = s < a[i];
        uint64_t s2 = s + carry;
        uint64_t c2 = s2 < s;
        r[i] = s2;
        carry = c1 | c2;
    }
}

__device__ __forceinline__ WideSum DecodeWide(const AccSpec &s, const uint64_t *w)
{
    // Side value = sum over k of word_k * 2^(32k) (each word is a sum of 32-bit chunks).
    const int n = s.kind == ACC_WSUM2 ? 2 : 4;
    uint64_t pos[3] = {0, 0, 0};
    uint64_t neg[3] = {0, 0, 0};
    for (int k = 0; k < n; ++k) {
        uint64_t a[3] = {0, 0, 0};
        uint64_t b[3] = {0, 0, 0};
        const int sh = 32 * k;
        const int wi = sh >> 6;
        const int bi = sh & 63;
        a[wi] = w[k] << bi;
        b[wi] = w[n + k] << bi;
        if (bi != 0 && wi + 1 < 3) {
            a[wi + 1] = w[k] >> (64 - bi);
            b[wi + 1] = w[n + k] >> (64 - bi);
        }
        Add192(pos, a, pos);
        Add192(neg, b, neg);
    }
    WideSum r;
    if (Cmp192(pos, neg) >= 0) {
        r.negative = false;
        Sub192(pos, neg, r.mag);
    } else {
        r.negative = true;
        Sub192(neg, pos, r.mag);
    }
    Add192(pos, neg, r.abs);
    return r;
}

// True if magnitude `m` (192-bit) exceeds the bound of the output: int64 range (negative
// sums may reach 2^63) or 10^38 - 1.
__device__ __forceinline__ bool ExceedsBound(const uint64_t *m, bool negative, int boundKind)
{
    if (boundKind == 0) {
        if (m[2] != 0 || m[1] != 0) {
            return true;
        }
        return negative ? (m[0] > 0x8000000000000000ull) : (m[0] > 0x7fffffffffffffffull);
    }
    if (m[2] != 0) {
        return true;
    }
    const unsigned __int128 v = (static_cast<unsigned __int128>(m[1]) << 64) | m[0];
    return v > Dec38Max();
}

// Whether an exact sum's sticky-overflow outcome is an overflow: the total beyond the bound
// always is; a total within it whose sum of magnitudes exceeds the bound depends on the row
// order and is decided by the ordered replay (the slot is queued for it, or its answer read).
__device__ __forceinline__ bool ExactSumOverflowed(const AggExtract &e, const OutSpec &os, const WideSum &ws,
    uint64_t s)
{
    bool overflow = ExceedsBound(ws.mag, ws.negative, os.boundKind);
    if (!overflow && ExceedsBound(ws.abs, false, os.boundKind)) {
        if (e.forcedOverflow != nullptr) {
            overflow = ((e.forcedOverflow[s] >> os.pad) & 1u) != 0;
        } else {
            unsigned long long k = atomicAdd(e.nAmbiguous, 1ull);
            if (k < e.ambiguousCap) {
                e.ambiguousSlots[k] = s;
            }
        }
    }
    return overflow;
}

__device__ __forceinline__ unsigned __int128 Pow10U128(int n)
{
    unsigned __int128 p = 1;
    for (int i = 0; i < n; ++i) {
        p *= 10;
    }
    return p;
}

// Spark's decimal average of a checked sum (magnitude `sum`, the sign applied by the caller)
// over `count` rows (CalcAvg, average_spark_decimal_aggregator.h:477-546): the quotient's scale
// is max(6, sumScale + 21) at precision sumPrec - sumScale + scale, cut back to 38 digits
// keeping the integer digits and at least min(scale, 6) fractional ones; the sum is rescaled to
// it (checked against 10^38 - 1), divided by the count rounding half away from zero, and
// rescaled to the output scale (multiplied, checked, or divided, rounded again).  Magnitudes
// round the same way as the signed values.  False on overflow.
__device__ __forceinline__ bool DecimalAverage(unsigned __int128 sum, uint64_t count, int sumPrec, int sumScale,
    int outScale, unsigned __int128 *out)
{
    int scale = sumScale + 21 > 6 ? sumScale + 21 : 6;
    const int prec = sumPrec - sumScale + scale;
    if (prec > 38) {
        const int intDigits = prec - scale;
        const int minScale = scale < 6 ? scale : 6;
        scale = 38 - intDigits > minScale ? 38 - intDigits : minScale;
    }
    const unsigned __int128 f = Pow10U128(scale - sumScale);
    if (sum != 0 && sum > Dec38Max() / f) {
        return false;
    }
    const unsigned __int128 dividend = sum * f;
    const unsigned __int128 avg = (dividend + count / 2) / count;
    const int diff = outScale - scale;
    if (diff >= 0) {
        const unsigned __int128 g = Pow10U128(diff);
        if (avg != 0 && avg > Dec38Max() / g) {
            return false;
        }
        *out = avg * g;
    } else {
        const unsigned __int128 g = Pow10U128(-diff);
        *out = (avg + g / 2) / g;
    }
    return true;
}

// A zero value at output row `pos` (a 16-byte column holds two words per row).
__device__ __forceinline__ void StoreZero(const OutSpec &os, uint64_t pos)
{
    if (os.outWidth == 16) {
        uint64_t *dst = static_cast<uint64_t *>(os.values) + 2 * pos;
        dst[0] = 0;
        dst[1] = 0;
    } else {
        StoreWidth(os.values, pos, os.outWidth, 0);
    }
}

// Output row `pos` of the group in slot s (occupied) of table t: keys, counts and aggregates.
__device__ __forceinline__ void WriteGroup(const AggExtract &e, const AggTable &t, uint64_t s, const uint64_t *slot,
    uint64_t pos)
{
    const uint64_t *st = slot + t.keyWords;
    const bool nullSlot = (s == t.capacity + kNullSlotOffset);
    const bool sentinelSlot = (s == t.capacity + kSentinelSlotOffset);
    for (int o = 0; o < e.nOut; ++o) {
        const OutSpec &os = e.out[o];
        if (os.kind == OUT_KEY) {
            const KeyCol &kc = e.key.cols[os.src];
            if (e.key.kind == KEY_SINGLE) {
                if (nullSlot) {
                    SetOutNull(os.nulls, pos);
                    StoreWidth(os.values, pos, os.outWidth, 0);
                } else {
                    StoreWidth(os.values, pos, os.outWidth, sentinelSlot ? kEmptyKey : slot[0]);
                }
            } else {
                const uint64_t *kwds = slot + 1;
                const uint32_t mask = static_cast<uint32_t>(
                    (kwds[e.key.maskByte >> 3] >> ((e.key.maskByte & 7) * 8)) & 0xffu);
                const bool isNull = (mask >> os.src) & 1u;
                const int wi = kc.byteOffset >> 3;
                if (kc.width == 16) {
                    uint64_t *dst = static_cast<uint64_t *>(os.values) + 2 * pos;
                    dst[0] = isNull ? 0 : kwds[wi];
                    dst[1] = isNull ? 0 : kwds[wi + 1];
                } else {
                    const int sh = (kc.byteOffset & 7) * 8;
                    uint64_t bits = kwds[wi] >> sh;
                    StoreWidth(os.values, pos, os.outWidth, isNull ? 0 : bits);
                }
                if (isNull) {
                    SetOutNull(os.nulls, pos);
                }
            }
            continue;
        }
        if (os.kind == OUT_COUNT_MERGE) {
            StoreWidth(os.values, pos, 8, st[e.accs[os.src].word]);
            continue;
        }
        // A merging stage's decimal SUM saw a NULL partial sum: that partial overflowed, and the
        // overflow is sticky whatever the row order (sum_spark_decimal_aggregator.h, final stage).
        const bool flagged = os.flagAcc > 0 && st[e.accs[os.flagAcc].word] != 0;
        if (os.kind == OUT_IS_EMPTY) {
            const int64_t n = static_cast<int64_t>(st[e.accs[0].word]) -
                static_cast<int64_t>(st[e.accs[os.countAcc].word]);
            StoreWidth(os.values, pos, 1, (n == 0 && !flagged) ? 1u : 0u);
            continue;
        }
        if (os.kind == OUT_AVG_MERGE || os.kind == OUT_AVG_PARTIAL_SUM) {
            const uint64_t *w = st + e.accs[os.src].word;
            double sum = __dadd_rn(__longlong_as_double(static_cast<long long>(w[0])),
                __longlong_as_double(static_cast<long long>(w[1])));
            if (!isfinite(__longlong_as_double(static_cast<long long>(w[0])))) {
                sum = __longlong_as_double(static_cast<long long>(w[0]));
            }
            int64_t n;
            if (os.kind == OUT_AVG_MERGE || os.boundKind == 1) {
                n = static_cast<int64_t>(st[e.accs[os.countAcc].word]);  // summed partial counts
            } else {
                n = static_cast<int64_t>(st[e.accs[0].word]) - static_cast<int64_t>(st[e.accs[os.countAcc].word]);
            }
            if (n == 0) {
                if (os.kind == OUT_AVG_MERGE) {
                    SetOutNull(os.nulls, pos);
                }
                static_cast<double *>(os.values)[pos] = 0.0;
            } else {
                static_cast<double *>(os.values)[pos] = os.kind == OUT_AVG_MERGE ? sum / static_cast<double>(n) : sum;
            }
            continue;
        }
        int64_t cnt = static_cast<int64_t>(st[e.accs[0].word]);  // accs[0] is COUNT_ALL
        if (os.countAcc >= 0) {
            cnt = os.countSummed ? static_cast<int64_t>(st[e.accs[os.countAcc].word])
                                 : cnt - static_cast<int64_t>(st[e.accs[os.countAcc].word]);
        }
        if (os.kind == OUT_COUNT) {
            StoreWidth(os.values, pos, 8, static_cast<uint64_t>(cnt));
            continue;
        }
        if (flagged || (cnt == 0 && os.partial != 0)) {
            // An overflowed merge: NULL (an error unless overflow is NULL or the output is a
            // partial).  An empty partial sum: 0, not NULL.
            if (flagged) {
                SetOutNull(os.nulls, pos);
                if (!e.overflowAsNull && os.partial != 1) {
                    SetError(e.error, 5);
                }
            }
            StoreZero(os, pos);
            continue;
        }
        if (cnt == 0) {
            SetOutNull(os.nulls, pos);
            StoreZero(os, pos);
            continue;
        }
        const AccSpec &acc = e.accs[os.src];
        const uint64_t *w = st + acc.word;
        switch (os.kind) {
            case OUT_SUM_WRAP:
            case OUT_MIN_INT:
            case OUT_MAX_INT:
            case OUT_STR_ID:  // a dictionary id; the host turns it back into the string
                StoreWidth(os.values, pos, os.outWidth, w[0]);
                break;
            case OUT_MINMAX_DEC128: {
                uint64_t *dst = static_cast<uint64_t *>(os.values) + 2 * pos;
                dst[0] = w[0];
                dst[1] = w[1];
                break;
            }
            case OUT_SUM_DOUBLE:
            case OUT_AVG: {
                double sum = __dadd_rn(__longlong_as_double(static_cast<long long>(w[0])),
                    __longlong_as_double(static_cast<long long>(w[1])));
                if (!isfinite(__longlong_as_double(static_cast<long long>(w[0])))) {
                    sum = __longlong_as_double(static_cast<long long>(w[0]));
                }
                const double v = (os.kind == OUT_AVG) ? sum / static_cast<double>(cnt) : sum;
                static_cast<double *>(os.values)[pos] = v;
                break;
            }
            case OUT_MIN_DOUBLE:
            case OUT_MAX_DOUBLE: {
                const double v = DoubleFromOrdered(static_cast<int64_t>(w[0]));
                if (os.outWidth == 4) {
                    static_cast<float *>(os.values)[pos] = static_cast<float>(v);
                } else {
                    static_cast<double *>(os.values)[pos] = v;
                }
                break;
            }
            case OUT_AVG_DEC: {
                WideSum ws = DecodeWide(acc, w);
                bool overflow = ExactSumOverflowed(e, os, ws, s);
                unsigned __int128 mag = 0;
                if (!overflow) {
                    const unsigned __int128 sum = (static_cast<unsigned __int128>(ws.mag[1]) << 64) | ws.mag[0];
                    overflow = !DecimalAverage(sum, static_cast<uint64_t>(cnt), os.sumPrec, os.sumScale, os.rescalePow,
                        &mag);
                }
                if (overflow) {
                    SetOutNull(os.nulls, pos);
                    if (!e.overflowAsNull) {
                        SetError(e.error, 5);
                    }
                    StoreZero(os, pos);
                    break;
                }
                const unsigned __int128 v = ws.negative ? (~mag + 1) : mag;
                if (os.outWidth == 16) {
                    uint64_t *dst = static_cast<uint64_t *>(os.values) + 2 * pos;
                    dst[0] = static_cast<uint64_t>(v);
                    dst[1] = static_cast<uint64_t>(v >> 64);
                } else {
                    StoreWidth(os.values, pos, os.outWidth, static_cast<uint64_t>(v));  // cut to 64 bits
                }
                break;
            }
            case OUT_SUM_EXACT: {
                WideSum ws = DecodeWide(acc, w);
                bool overflow = ExactSumOverflowed(e, os, ws, s);
                unsigned __int128 mag = (static_cast<unsigned __int128>(ws.mag[1]) << 64) | ws.mag[0];
                if (!overflow && os.rescalePow > 0) {
                    unsigned __int128 f = 1;
                    for (int i = 0; i < os.rescalePow; ++i) {
                        f *= 10;
                    }
                    // |mag| <= 10^38 - 1 < 2^127 and f <= 10^38: check mag * f <= bound.
                    if (mag != 0 && mag > Dec38Max() / f) {
                        overflow = true;
                    } else {
                        mag *= f;
                    }
                }
                if (overflow) {
                    SetOutNull(os.nulls, pos);
                    if (!e.overflowAsNull && os.partial != 1) {
                        SetError(e.error, 5);
                    }
                    mag = 0;
                }
                unsigned __int128 v = ws.negative ? (~mag + 1) : mag;
                if (os.outWidth == 16) {
                    uint64_t *dst = static_cast<uint64_t *>(os.values) + 2 * pos;
                    dst[0] = static_cast<uint64_t>(v);
                    dst[1] = static_cast<uint64_t>(v >> 64);
                } else {
                    StoreWidth(os.values, pos, os.outWidth, static_cast<uint64_t>(v));
                }
                break;
            }
            default:
                break;
        }
    }
}

}  // namespace
}  // namespace omg
