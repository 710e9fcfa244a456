"""Sums in the shared tables of the partitioned strategy, whose 64-bit words are added to in 32-bit halves:
carries, borrows and mixed signs, hot and spread groups, ragged tiles, NULLs; exact in numpy."""
import math

import numpy as np
import pytest

import omnioperator_gb300 as omg
from helpers import run_agg

pytestmark = pytest.mark.gpu

S, I, L, D = omg.ShortType(), omg.IntType(), omg.LongType(), omg.DoubleType()
SUM, CALL, MIN = omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_ALL, omg.OMNI_AGGREGATION_TYPE_MIN


@pytest.mark.parametrize("groups,rows", [(1, 9001), (3, 4097), (300, 50_001), (5000, 120_003)])
@pytest.mark.parametrize("sign", [0, 1, -1])
def test_word_sums_in_halves(gpu, groups, rows, sign):
    rng = np.random.default_rng(groups + sign)
    key = rng.integers(0, groups, rows)
    s = rng.integers(-2**15, 2**15, rows).astype(np.int16)
    i = rng.integers(-2**31, 2**31, rows).astype(np.int32)
    # Near multiples of 2^32 on both sides: low halves that carry with nearly every addition.
    v = rng.integers(-2**10, 2**10, rows) * 2**32 + rng.integers(-2, 3, rows)
    if sign:
        s, i, v = [(np.abs(x.astype(np.int64)) * sign) for x in (s, i, v)]
        s, i = np.clip(s, -2**15, 2**15 - 1).astype(np.int16), np.clip(i, -2**31, 2**31 - 1).astype(np.int32)
    d = rng.standard_normal(rows) * 10.0 ** rng.integers(-8, 9, rows)
    nulls = [None, rng.random(rows) < 0.1, None, rng.random(rows) < 0.1, rng.random(rows) < 0.1]
    cols, _ = run_agg([0], [L], [[1], [2], [3], [3], [4], []], [[S], [I], [L], [L], [D], []],
                      [[L], [L], [L], [L], [D], [L]], [SUM, SUM, SUM, MIN, SUM, CALL], [key, s, i, v, d],
                      [L, S, I, L, D], nulls=nulls, strategy=omg.AGG_STRATEGY_PARTITIONED, batch_sizes=(4096, 1000, 7))
    order = np.argsort(cols[0][0])
    uniq, inv = np.unique(key, return_inverse=True)
    assert np.array_equal(cols[0][0][order], uniq)
    for col, x, m in ((1, s, nulls[1]), (2, i, None), (3, v, nulls[3])):
        live = np.ones(rows, bool) if m is None else ~m
        want = np.zeros(len(uniq), np.int64)
        np.add.at(want, inv[live], x[live].astype(np.int64))
        some = np.bincount(inv[live], minlength=len(uniq)) > 0
        assert np.array_equal(~cols[col][1][order], some)
        assert np.array_equal(cols[col][0][order][some], want[some])
    live = ~nulls[3]
    low = np.full(len(uniq), np.iinfo(np.int64).max)
    np.minimum.at(low, inv[live], v[live])
    some = np.bincount(inv[live], minlength=len(uniq)) > 0
    assert np.array_equal(cols[4][0][order][some], low[some])
    assert np.array_equal(cols[6][0][order], np.bincount(inv, minlength=len(uniq)))
    # The first 64 rows of a table slot are added plainly, the later ones compensated: at most two slots' 64
    # additions of 2^-53 and one rounding of the result.
    live = ~nulls[4]
    for g in range(min(len(uniq), 50)):
        x = d[live & (inv == g)]
        if len(x):
            assert abs(cols[5][0][order][g] - math.fsum(x)) <= 130 * 2.0**-53 * np.abs(x).sum()


@pytest.mark.parametrize("keys", [1, 2])
@pytest.mark.parametrize("share", [0.02, 0.3, 0.95])
@pytest.mark.parametrize("groups", [500, 9000])
def test_hot_groups_with_double_sums(gpu, keys, share, groups):
    """Groups that fit the partitions, some of whose rows are one key's (or the NULL key's): AUTO takes the
    partitions or the radix passes, by the share of the hottest key and the width of the key."""
    rng = np.random.default_rng(groups + keys)
    rows = 400_003
    key = rng.integers(0, groups, rows)
    hot = rng.random(rows)
    key[hot < share] = 3
    km = hot < share / 3
    v = rng.integers(-2**40, 2**40, rows)
    d = rng.standard_normal(rows)
    dm = rng.random(rows) < 0.05
    kcols, ktypes = ([key], [L]) if keys == 1 else ([key, (key % 7).astype(np.int32)], [L, I])
    k = len(kcols)
    cols, _ = run_agg(list(range(k)), ktypes, [[k], [k + 1], [k + 1], []], [[L], [D], [D], []], [[L], [D], [D], [L]],
                      [SUM, SUM, MIN, CALL], kcols + [v, d], ktypes + [L, D],
                      nulls=[km] + [None] * k + [dm], batch_sizes=(100_000, 4096))
    code = np.where(km, groups + (key % 7 if keys == 2 else 0), key)
    uniq, inv = np.unique(code, return_inverse=True)
    got = np.where(cols[0][1], groups + (cols[1][0] if keys == 2 else 0), cols[0][0])
    order = np.argsort(got)
    assert np.array_equal(got[order], uniq)
    want = np.zeros(len(uniq), np.int64)
    np.add.at(want, inv, v)
    assert np.array_equal(cols[k][0][order], want)
    low = np.full(len(uniq), np.inf)
    np.minimum.at(low, inv[~dm], d[~dm])
    some = np.bincount(inv[~dm], minlength=len(uniq)) > 0
    assert np.array_equal(cols[k + 2][0][order][some], low[some])
    assert np.array_equal(cols[k + 3][0][order], np.bincount(inv, minlength=len(uniq)))
    mass = np.bincount(inv[~dm], weights=np.abs(d[~dm]), minlength=len(uniq))
    for g in list(range(0, len(uniq), 97)) + [3, len(uniq) - 1]:
        # Each partial table leaves at most 64 plain additions of its own rows: 64 * 2^-53 of the group's mass.
        exact = math.fsum(d[~dm & (inv == g)])
        assert abs(cols[k + 1][0][order][g] - exact) <= 66 * 2.0**-53 * mass[g]
