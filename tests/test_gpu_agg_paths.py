"""Which kernels AUTO takes, and that they give what the global table gives, over the forms of input that each of them
accepts: every type, NULLs, masks, strings, infinities and NaN, hot groups, tables that are too small."""
import ctypes

import numpy as np
import pytest

import omnioperator_gb300 as omg
from helpers import run_agg

pytestmark = pytest.mark.gpu

S, I, L, D, F = omg.ShortType(), omg.IntType(), omg.LongType(), omg.DoubleType(), omg.DataType(omg.OMNI_FLOAT)
D64, D128, V, B = omg.Decimal64Type(18, 2), omg.Decimal128Type(38, 2), omg.VarcharType(24), omg.BooleanType()
SUM, CNT, CALL, AVG, MAX, MIN = (omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_COLUMN,
                                 omg.OMNI_AGGREGATION_TYPE_COUNT_ALL, omg.OMNI_AGGREGATION_TYPE_AVG,
                                 omg.OMNI_AGGREGATION_TYPE_MAX, omg.OMNI_AGGREGATION_TYPE_MIN)
TABLE, PARTITIONS, FEW, RADIX, SMALL = 1, 2, 3, 4, 5


def last_kernel():
    """(kernel, passes over a partition, units of hot partitions, whole partitions)"""
    out = (ctypes.c_int64 * 4)()
    omg.check(omg.lib().omg_debug_last_agg_kernel(out, 4))
    return tuple(out)


# Plans: (function, column of the value columns below, input type, output type, masked)
PLANS = {
    "doubles": [(SUM, "d", D, D, 0), (MIN, "d", D, D, 0), (AVG, "f", F, D, 0), (MAX, "f", F, F, 0)],
    "whole": [(SUM, "s", S, L, 0), (MIN, "i", I, I, 0), (MAX, "l", L, L, 0), (SUM, "l", L, L, 0), (CNT, "i", I, L, 0),
              (SUM, "x", D64, D128, 0)],
    "wide": [(SUM, "w", D128, D128, 0), (MIN, "w", D128, D128, 0), (MAX, "w", D128, D128, 0), (CNT, "w", D128, L, 0)],
    "strings": [(MIN, "v", V, V, 0), (MAX, "v", V, V, 0), (CNT, "v", V, L, 0), (CALL, None, None, L, 0)],
    "masks": [(SUM, "l", L, L, 1), (CALL, None, None, L, 1), (MIN, "d", D, D, 1), (SUM, "l", L, L, 0)],
}
TYPES = {"s": S, "i": I, "l": L, "d": D, "f": F, "x": D64, "w": D128, "v": V, "m": B}


def _columns(code, n, rng):
    """Doubles are whole numbers, whose sums are exact in any order; one group in three has an infinity, one both,
    one a NaN."""
    d = rng.integers(-2**30, 2**30, n).astype(np.float64)
    f = rng.integers(-2**20, 2**20, n).astype(np.float32)
    for x in (d, f):
        odd = rng.random(n) < 0.2
        x[odd & (code % 7 == 1)] = np.inf
        x[odd & (code % 7 == 2)] = -np.inf
        x[odd & (code % 7 == 3)] = np.where(rng.random(int((odd & (code % 7 == 3)).sum())) < 0.5, np.inf, -np.inf)
        x[odd & (code % 7 == 4)] = np.nan
        x[code % 1009 == 5] = np.nan
        x[code % 1009 == 6] = -0.0
    w = np.stack([rng.integers(0, 2**63, n).astype(np.uint64), np.zeros(n, np.uint64)], axis=1)
    neg = rng.random(n) < 0.4
    w[neg, 1] = np.uint64(2**64 - 1)
    words = np.array([b"%05d" % (k * 7919 % 100_000) + b"\xff" * (k % 3) for k in range(2000)], dtype=object)
    return {"s": rng.integers(-2**15, 2**15, n).astype(np.int16), "i": rng.integers(-2**31, 2**31, n).astype(np.int32),
            "l": rng.integers(-2**60, 2**60, n), "d": d, "f": f, "x": rng.integers(-10**17, 10**17, n), "w": w,
            "v": words[rng.integers(0, 2000, n)], "m": (rng.random(n) < 0.6).astype(np.int8)}


def _sorted_rows(cols, nkeys):
    order = np.lexsort([x for v, m in cols[:nkeys] for x in (np.where(m, 0, v), m)])
    return [(v[order], np.asarray(m)[order]) for v, m in cols]


def _same(a, b):
    if a.dtype.kind == "f":
        return np.array_equal(a.view(f"i{a.itemsize}")[~np.isnan(a)], b.view(f"i{b.itemsize}")[~np.isnan(b)]) and \
            np.array_equal(np.isnan(a), np.isnan(b))
    return np.array_equal(a, b)


def _keys(kind, code, rng):
    km = rng.random(len(code)) < 0.01
    if kind == "long":
        key = code * 2**40 - 12345
        key[code == 1] = np.iinfo(np.int64).min
        return [key], [L], [km]
    return [(code % 13).astype(np.int32), code * 2**33], [I, L], [km, None]


def _compare(code, key_kind, plan, batch_sizes, seed, **auto):
    """AUTO against the global table; AUTO's kernel."""
    rng = np.random.default_rng(seed)
    n = len(code)
    keys, ktypes, kmasks = _keys(key_kind, code, rng)
    data = _columns(code, n, rng)
    spec = PLANS[plan]
    used = list(dict.fromkeys([c for _, c, _, _, _ in spec if c is not None])) + ["m"]
    nulls = [(rng.random(n) < 0.05) if c != "m" else (rng.random(n) < 0.1) for c in used]
    at = {c: len(keys) + i for i, c in enumerate(used)}
    args = dict(group_cols=list(range(len(keys))), group_types=ktypes,
                aggs_cols=[[] if c is None else [at[c]] for _, c, _, _, _ in spec],
                agg_in_types=[[] if t is None else [t] for _, _, t, _, _ in spec], agg_out_types=[[o] for *_, o, _ in spec],
                funcs=[f for f, *_ in spec], columns=keys + [data[c] for c in used],
                types=ktypes + [TYPES[c] for c in used], nulls=kmasks + nulls, overflow_as_null=True,
                mask_cols=[at["m"] if masked else 0xFFFFFFFF for *_, masked in spec])
    got, _ = run_agg(**args, batch_sizes=batch_sizes, **auto)
    kernel = last_kernel()
    want, _ = run_agg(**args, batch_sizes=(n,), strategy=omg.AGG_STRATEGY_GLOBAL)
    assert last_kernel()[0] == TABLE
    got, want = _sorted_rows(got, len(keys)), _sorted_rows(want, len(keys))
    for c, ((gv, gm), (wv, wm)) in enumerate(zip(got, want)):
        assert np.array_equal(gm, wm), c
        live = ~np.asarray(gm, dtype=bool)
        assert _same(gv[live], wv[live]), c
    return kernel


@pytest.mark.parametrize("key", ["long", "pair"])
@pytest.mark.parametrize("plan,kernel", [("doubles", FEW), ("whole", FEW), ("masks", FEW), ("wide", PARTITIONS),
                                         ("strings", PARTITIONS)])
def test_few_groups(gpu, key, plan, kernel):
    """Groups with their states in every thread; decimal128 and string states have no such form."""
    code = np.random.default_rng(1).integers(1, 4, 280_003)
    assert _compare(code, key, plan, (100_000, 777), 2)[0] == kernel


@pytest.mark.parametrize("key", ["long", "pair"])
@pytest.mark.parametrize("plan", PLANS)
def test_radix_passes(gpu, key, plan):
    """More groups than the partitions hold, a fifth of the rows one group's (its partition is cut into units)."""
    rng = np.random.default_rng(3)
    n = 700_003
    code = rng.integers(0, 3_000_000, n)
    code[rng.random(n) < 0.2] = 4321
    kernel, passes, cut, whole = _compare(code, key, plan, (120_000, 999), 4, strategy=omg.AGG_STRATEGY_AUTO,
                                          capacity_hint=600_000)
    assert (kernel, passes) == (RADIX, 1) and cut > 1 and whole > 1


@pytest.mark.parametrize("key", ["long", "pair"])
@pytest.mark.parametrize("plan", ["doubles", "whole", "wide"])
def test_small_calls(gpu, key, plan):
    code = np.random.default_rng(5).integers(0, 300, 6_000)
    assert _compare(code, key, plan, (3000, 1700), 6)[0] == SMALL


@pytest.mark.parametrize("key", ["long", "pair"])
@pytest.mark.parametrize("plan", PLANS)
def test_partitions(gpu, key, plan):
    code = np.random.default_rng(7).integers(0, 2_000, 270_000)
    assert _compare(code, key, plan, (100_000,), 8)[0] == PARTITIONS


def test_several_passes_over_a_partition(gpu):
    """Five decimal128 sums, some 350 bytes a group: 2^14 partitions hold three and a half million groups."""
    n = 4_000_000
    key = np.random.default_rng(9).permutation(n).astype(np.int64) * 7919
    vals = np.zeros((n, 2), np.uint64)
    vals[:, 0] = np.arange(n, dtype=np.uint64) + 1
    cols, _ = run_agg([0], [L], [[c] for c in range(1, 6)], [[D128]] * 5, [[D128]] * 5, [SUM] * 5,
                      [key] + [vals] * 5, [L] + [D128] * 5, batch_sizes=(n,))
    kernel, passes, _, whole = last_kernel()
    assert kernel == RADIX and passes > 1 and whole > 1
    order, want = np.argsort(cols[0][0], kind="stable"), np.argsort(key, kind="stable")
    assert np.array_equal(cols[0][0][order], key[want])
    for v, m in cols[1:]:
        assert not m.any() and np.array_equal(v[order], vals[want])


@pytest.mark.parametrize("keys,groups,rows,share,kernel", [
    (1, 500, 400_003, 0.02, PARTITIONS), (1, 500, 400_003, 0.95, RADIX),
    (2, 2000, (1 << 21) - 1, 0.0, PARTITIONS), (2, 2000, 1 << 21, 0.0, RADIX), (2, 300, 1 << 21, 0.0, PARTITIONS),
    (2, 1000, 1 << 21, 0.0, PARTITIONS)])  # (0.27 of a table's 3,657 slots; 2,000 groups 0.55)
def test_groups_that_fit_the_partitions(gpu, keys, groups, rows, share, kernel):
    """With sums of doubles the radix passes take hot groups, and wide keys of many rows and groups."""
    rng = np.random.default_rng(rows + groups)
    key = rng.integers(0, groups, rows)
    key[rng.random(rows) < share] = 3
    d = rng.integers(-2**30, 2**30, rows).astype(np.float64)
    kcols, ktypes = ([key], [L]) if keys == 1 else ([key, (key % 7).astype(np.int32)], [L, I])
    k = len(kcols)
    cols, _ = run_agg(list(range(k)), ktypes, [[k], []], [[D], []], [[D], [L]], [SUM, CALL], kcols + [d], ktypes + [D],
                      batch_sizes=(rows,))
    assert last_kernel()[0] == kernel
    order = np.argsort(cols[0][0])
    assert np.array_equal(cols[k][0][order], np.bincount(key, weights=d, minlength=groups))
    assert np.array_equal(cols[k + 1][0][order], np.bincount(key, minlength=groups))


def _unmix(h):
    """The key whose hash is h: the hash's steps undone."""
    h = h ^ (h >> np.uint64(33))
    h = h * np.uint64(pow(0xC4CEB9FE1A85EC53, -1, 2**64))
    h = h ^ (h >> np.uint64(33))
    h = h * np.uint64(pow(0xFF51AFD7ED558CCD, -1, 2**64))
    return (h ^ (h >> np.uint64(33))).view(np.int64)


@pytest.mark.parametrize("copies", [1, 30])
def test_radix_tables_that_overflow(gpu, copies):
    """3,000 keys of one partition, more than its table holds, that start at the same slot of the global table, too:
    single rows (the records queue up and are run again) or 30 each (units' tables whose groups find no slot are
    kept and merged) after the global table has grown."""
    rng = np.random.default_rng(11)
    m = 3000
    low = np.uint64(0x123456) << np.uint64(18) & np.uint64(0xFFFFFFFF)  # the partition's bits
    h = (np.arange(1, m + 1, dtype=np.uint64) * np.uint64(1_234_567) << np.uint64(32)) | low | \
        (rng.integers(0, 256, m).astype(np.uint64) << np.uint64(10)) | np.uint64(77)
    crafted = _unmix(h)
    key = np.concatenate([np.repeat(crafted, copies), rng.integers(-2**62, 2**62, 400_000)])
    key = key[rng.permutation(len(key))]
    v = rng.integers(-2**40, 2**40, len(key))
    d = rng.integers(-2**30, 2**30, len(key)).astype(np.float64)
    cols, ctr = run_agg([0], [L], [[1], [2], [2]], [[L], [D], [D]], [[L], [D], [D]], [SUM, SUM, MAX], [key, v, d], [L, L, D],
                        batch_sizes=(len(key),))
    kernel, _, cut, _ = last_kernel()
    assert kernel == RADIX and (cut > 0) == (copies > 1)
    assert ctr["resizes"] >= 1 and (copies > 1 or ctr["retried_rows"] > 0)
    uniq, inv = np.unique(key, return_inverse=True)
    order = np.argsort(cols[0][0])
    assert np.array_equal(cols[0][0][order], uniq)
    want, top = np.zeros(len(uniq), np.int64), np.full(len(uniq), -np.inf)
    np.add.at(want, inv, v)
    np.maximum.at(top, inv, d)
    assert np.array_equal(cols[1][0][order], want)
    assert np.array_equal(cols[2][0][order], np.bincount(inv, weights=d, minlength=len(uniq)))
    assert np.array_equal(cols[3][0][order], top)


@pytest.mark.parametrize("key", ["long", "pair"])
@pytest.mark.parametrize("plan,groups,kernel", [
    ("six", 9, FEW), ("six", 10, FEW), ("six", 12, FEW), ("six", 13, PARTITIONS),
    ("sum", 21, FEW), ("sum", 22, FEW), ("sum", 29, FEW), ("sum", 34, FEW), ("sum", 40, PARTITIONS)])
def test_few_groups_up_to_the_most(gpu, key, plan, groups, kernel):
    """Up to what 256 threads have room for without the errors of the double sums; with them the most groups take 192
    threads (six aggregates from 10, one sum from 22) and 128 (one sum from 29)."""
    rng = np.random.default_rng(groups)
    n = 270_001
    code = rng.integers(0, groups, n)
    keys, ktypes = ([code * 2**40], [L]) if key == "long" else ([(code % 13).astype(np.int32), code * 2**33], [I, L])
    k = len(keys)
    v = rng.integers(-2**40, 2**40, n)
    d = rng.integers(-2**30, 2**30, n).astype(np.float64)
    spec = [(SUM, k, L, L), (CNT, k, L, L), (MIN, k, L, L), (MAX, k, L, L), (SUM, k + 1, D, D), (AVG, k + 1, D, D)]
    spec = spec if plan == "six" else spec[4:5]
    cols, _ = run_agg(list(range(k)), ktypes, [[c] for _, c, _, _ in spec], [[t] for _, _, t, _ in spec],
                      [[o] for *_, o in spec], [f for f, *_ in spec], keys + [v, d], ktypes + [L, D], batch_sizes=(100_000,))
    assert last_kernel()[0] == kernel
    order = np.argsort(cols[k - 1][0])
    count = np.bincount(code, minlength=groups)
    total = np.bincount(code, weights=d, minlength=groups)
    lo, hi = np.full(groups, 2**60), np.full(groups, -2**60)
    np.minimum.at(lo, code, v)
    np.maximum.at(hi, code, v)
    want = {"six": [np.bincount(code, weights=v, minlength=groups).astype(np.int64), count, lo, hi, total, total / count],
            "sum": [total]}[plan]
    if plan == "six":
        want[0] = np.zeros(groups, np.int64)
        np.add.at(want[0], code, v)
    assert len(order) == groups
    for (got, _), w in zip(cols[k:], want):
        assert np.array_equal(got[order], w)
