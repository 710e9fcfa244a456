"""What the operators ask of device and pinned memory: a path that wants more must not turn a call away that fits another,
and results must not hold much more than their rows."""
import ctypes

import numpy as np
import pytest

import omnioperator_gb300 as omg
from helpers import run_agg

pytestmark = pytest.mark.gpu

L, I, D, V = omg.LongType(), omg.IntType(), omg.DoubleType(), omg.VarcharType(24)
SUM, CNT, CALL = (omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_COLUMN,
                  omg.OMNI_AGGREGATION_TYPE_COUNT_ALL)
MB = 1 << 20


def memory():
    """(device bytes held, the most since the latest call, pinned bytes held)"""
    out = (ctypes.c_int64 * 3)()
    omg.check(omg.lib().omg_debug_memory(out, 3))
    return tuple(out)


def last_agg_kernel():
    out = (ctypes.c_int64 * 4)()
    omg.check(omg.lib().omg_debug_last_agg_kernel(out, 4))
    return out[0]


def _sums(key, v, strategy, hint, limit=0):
    """SUM and COUNT by key: (sorted keys, their sums, peak of device memory above what was held before)."""
    fac = omg.HashAggregationOperatorFactory([0], [L], [[1], [1]], [[L], [L]], [[L], [L]], [SUM, CNT])
    host = omg.make_batch([L, L], [key, v])
    batch = omg.batch_to_device(host)
    omg.free_batch(host)
    op = fac.create_operator()
    try:
        op.set_agg_strategy(strategy, hint)
        before = memory()[0]
        op.add_input(batch)
        omg.lib().omg_debug_limit_device_memory(before + limit if limit else 0)
        outs = op.drain()
        omg.lib().omg_debug_limit_device_memory(0)
        peak = memory()[1] - before
        parts = [omg.batch_to_numpy(b) for b in outs]
        omg.free_batches(outs)
    finally:
        omg.lib().omg_debug_limit_device_memory(0)
        op.delete()
        fac.close()
    keys, sums = (np.concatenate([p[c][0] for p in parts]) for c in (0, 1))
    order = np.argsort(keys)
    return keys[order], sums[order], peak


def test_radix_passes_without_the_memory_for_them(gpu):
    """Limits from what the global table takes up to what the radix passes take, so that each of their allocations is
    the one that fails: the call goes through all the same."""
    rng = np.random.default_rng(1)
    key = rng.integers(0, 400_000, 2_000_000) * 7919
    v = rng.integers(-2**40, 2**40, len(key))
    want = _sums(key, v, omg.AGG_STRATEGY_GLOBAL, 400_000)
    free = _sums(key, v, omg.AGG_STRATEGY_AUTO, 400_000)
    assert last_agg_kernel() == 4 and free[2] > want[2] + 4 * MB
    kernels = set()
    for limit in np.linspace(want[2] + MB, free[2] - 1, 12).astype(int):
        got = _sums(key, v, omg.AGG_STRATEGY_AUTO, 400_000, int(limit))
        kernels.add(last_agg_kernel())
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert kernels == {1}
    assert np.array_equal(free[0], want[0]) and np.array_equal(free[1], want[1])


@pytest.mark.parametrize("budget", [40 * MB, 200 * MB])
def test_budgeted_aggregations_take_no_radix_passes(gpu, budget):
    """A budget is for the group table (64 MB here): neither the partitions of a spilled run nor a run that fits are
    aggregated by passes that hold the rows and the groups once more."""
    rng = np.random.default_rng(2)
    n = 2_000_000
    key = rng.integers(0, 1_000_000, n) * 7919
    v = rng.integers(-2**40, 2**40, n)
    cols, _ = run_agg([0], [L], [[1], [1]], [[L], [L]], [[L], [L]], [SUM, CNT], [key, v], [L, L], batch_sizes=(n,),
                      spill_budget=budget)
    assert last_agg_kernel() != 4
    order = np.argsort(cols[0][0])
    uniq, inv = np.unique(key, return_inverse=True)
    want = np.zeros(len(uniq), np.int64)
    np.add.at(want, inv, v)
    assert np.array_equal(cols[0][0][order], uniq) and np.array_equal(cols[1][0][order], want)


def test_more_rows_after_a_radix_flush(gpu):
    """The groups of the first rows move into a table of the size that an exact estimate would have given it."""
    n, groups = 500_000, 260_000
    key = np.arange(n, dtype=np.int64) % groups * 7919
    slots = 1 << 19  # the least power of two that is at least twice the groups
    slot_bytes = 8 * 4  # key, COUNT(*), NULLs, sum
    fac = omg.HashAggregationOperatorFactory([0], [L], [[1], [1]], [[L], [L]], [[L], [L]], [SUM, CNT])
    op = fac.create_operator()
    try:
        op.set_agg_strategy(omg.AGG_STRATEGY_AUTO, groups)
        omg.lib().omg_debug_set_agg_flush_rows(n)
        before = memory()[0]
        for k in range(2):
            op.add_input(omg.make_batch([L, L], [key, np.full(n, k + 1)]))
            assert last_agg_kernel() == (4, 1)[k]
        assert memory()[0] - before <= (slots + 2) * slot_bytes + MB
        outs = op.drain()
        cols = [omg.batch_to_numpy(b) for b in outs]
        omg.free_batches(outs)
    finally:
        omg.lib().omg_debug_set_agg_flush_rows(0)
        op.delete()
        fac.close()
    got = np.concatenate([c[0][0] for c in cols])
    order = np.argsort(got)
    assert np.array_equal(got[order], np.unique(key))
    assert np.array_equal(np.concatenate([c[1][0] for c in cols])[order], 3 * np.bincount(key // 7919))


def _join(bkey, pay, ptype, pkey, batch=None, device=True, limit=0, filt=None, kind=omg.OMNI_JOIN_TYPE_INNER, state=None):
    """Rows (key, payload) of the join and what memory it took: (rows sorted, device bytes held by the outputs, peak,
    counters, pinned bytes held by the outputs)."""
    bf = omg.HashBuilderOperatorFactory(kind, [L, ptype], [0])
    bop = bf.create_operator()
    bop.add_input(omg.make_batch([L, ptype], [bkey, pay]))
    bop.get_output()
    pf = omg.LookupJoinOperatorFactory([L], [0], [0], [1], [ptype], bf, filter_expr=filt)
    op = pf.create_operator()
    try:
        op.set_device_output(device)
        host = omg.make_batch([L], [pkey])
        b = omg.batch_to_device(host)
        omg.free_batch(host)
        before = memory()
        omg.lib().omg_debug_limit_device_memory(before[0] + limit if limit else 0)
        op.add_input(b)
        outs = op.drain()
        ctr = op.counters()
        after = memory()
        omg.lib().omg_debug_limit_device_memory(0)
        parts = []
        for o in outs:
            h = omg.batch_to_host(o) if device else o
            parts.append(omg.batch_to_numpy(h))
            if device:
                omg.free_batch(h)
        omg.free_batches(outs)
    finally:
        omg.lib().omg_debug_limit_device_memory(0)
        op.delete()
        pf.close()
        bop.delete()
        bf.close()
    keys, vals = (np.concatenate([p[c][0] for p in parts]) if parts else np.zeros(0, np.int64) for c in (0, 1))
    order = np.lexsort([vals, keys])
    return keys[order], vals[order], after[0] - before[0], after[1] - before[0], ctr, after[2] - before[2]


def _joined(bkey, pay, pkey):
    order = np.argsort(bkey, kind="stable")
    lo, hi = np.searchsorted(bkey[order], pkey, "left"), np.searchsorted(bkey[order], pkey, "right")
    n = hi - lo
    rows = np.repeat(lo, n) + np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n)
    keys, vals = np.repeat(pkey, n), pay[order][rows]
    order = np.lexsort([vals, keys])
    return keys[order], vals[order]


def _hot_build():
    """One key of 1,000 rows, 64,000 of one row."""
    bkey = np.concatenate([np.arange(64_000), np.full(999, 77)]) * 1_000_003
    return bkey, np.arange(len(bkey), dtype=np.int32)


@pytest.mark.parametrize("hot", [0, 300])
def test_join_reserves_for_the_mean_of_a_key(gpu, hot):
    """65,536 probe rows, of which none or 300 are of the key with 1,000 rows: rooms for 1,000 rows each would be
    786 MB.  Where the hot key overflows them the probe runs once more at the exact size."""
    bkey, pay = _hot_build()
    pkey = (np.random.default_rng(3).integers(100, 64_000, 65_536)) * 1_000_003
    pkey[:hot] = 77 * 1_000_003
    keys, vals, held, peak, ctr, _ = _join(bkey, pay, I, pkey)
    want = _joined(bkey, pay, pkey)
    assert np.array_equal(keys, want[0]) and np.array_equal(vals, want[1])
    assert ctr["resizes"] == (1 if hot else 0)
    if not hot:
        assert held <= 2 * len(pkey) * 12 + 2 * MB and peak <= 4 * len(pkey) * 12 + 2 * MB


def _few_hits(varchar):
    """2,000 keys of 50 rows each, and 65,536 probe rows of which one in a hundred has a match."""
    rng = np.random.default_rng(4)
    bkey = np.repeat(np.arange(2000), 50) * 1_000_003
    pay = np.arange(len(bkey), dtype=np.int32)
    if varchar:
        pay = np.array([b"%05d" % p for p in pay], dtype=object)
    pkey = np.where(rng.random(65_536) < 0.01, rng.integers(0, 2000, 65_536), 5000 + rng.integers(0, 2000, 65_536))
    return bkey, pay, pkey * 1_000_003


@pytest.mark.parametrize("device", [False, True])
def test_strings_of_a_join_are_built_over_two_rows_a_probe_row(gpu, device):
    """Not over the 50 rows that a key has: row numbers, lengths, two kinds of offsets, 24 bytes a position."""
    bkey, pay, pkey = _few_hits(True)
    keys, vals, _, peak, _, _ = _join(bkey, pay, V, pkey, device=device)
    want = _joined(bkey, pay, pkey)
    assert np.array_equal(keys, want[0]) and np.array_equal(vals, want[1])
    assert peak <= 2 * len(pkey) * (8 + 24) + 2 * MB


@pytest.mark.parametrize("kind", [omg.OMNI_JOIN_TYPE_INNER, omg.OMNI_JOIN_TYPE_LEFT])
@pytest.mark.parametrize("device,limit", [(True, 0), (True, 12 * MB), (False, 0)])
def test_joins_that_come_to_less_than_the_mean(gpu, device, limit, kind):
    """The output holds about what it needs, not 56 rows a probe row (44 MB), which the probe can do without, too."""
    bkey, pay, pkey = _few_hits(False)
    keys, vals, held, _, ctr, pinned = _join(bkey, pay, I, pkey, device=device, limit=limit, kind=kind)
    want = _joined(bkey, pay, pkey)
    if kind == omg.OMNI_JOIN_TYPE_LEFT:
        miss = pkey[pkey >= 5000 * 1_000_003]
        want = np.concatenate([want[0], miss]), np.concatenate([want[1], np.zeros(len(miss), np.int32)])
        order = np.lexsort([want[1], want[0]])
        want = want[0][order], want[1][order]
    assert np.array_equal(keys, want[0])
    hits = keys < 2000 * 1_000_003
    assert np.array_equal(vals[hits], want[1][hits])
    assert ctr["resizes"] == 0
    assert (held if device else pinned) <= 2 * len(pkey) * 13 + 2 * MB


@pytest.mark.parametrize("filtered,limit", [(True, 0), (False, 2 * MB)])
def test_payload_of_duplicates_only_where_it_is_read_and_fits(gpu, filtered, limit):
    """The build side's payload in key order, 3.2 MB here: not for a join with a filter, whose kernel does not read it,
    and not a reason for a probe to fail."""
    bkey = np.repeat(np.arange(200_000), 2) * 1_000_003
    pay = np.arange(len(bkey), dtype=np.int32) - 200_000
    pkey = np.random.default_rng(5).integers(0, 250_000, 4096) * 1_000_003
    filt = omg.Binary(omg.EXPR_GTE, omg.Field(2, I), omg.Literal(0, I)) if filtered else None
    keys, vals, held, *_ = _join(bkey, pay, I, pkey, filt=filt, limit=limit)
    want = _joined(bkey, pay, pkey)
    if filtered:
        want = want[0][want[1] >= 0], want[1][want[1] >= 0]
    assert np.array_equal(keys, want[0]) and np.array_equal(vals, want[1])
    assert held <= MB


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("rows", [5_000, 40_000, 300_000])
def test_aggregation_results_hold_about_their_rows(gpu, rows, device):
    """100 groups, for which up to a row per input row was reserved: 2 MB for 40,000 rows."""
    rng = np.random.default_rng(6)
    key = rng.integers(0, 100, rows)
    v, d = rng.integers(-100, 100, rows), rng.integers(-100, 100, rows).astype(np.float64)
    nulls = [None, rng.random(rows) < 0.5, (key % 3 == 0)]
    fac = omg.HashAggregationOperatorFactory([0], [L], [[1], [1], [2], []], [[L], [L], [D], []], [[L], [L], [D], [L]],
                                             [SUM, CNT, SUM, CALL])
    before = memory()
    op = fac.create_operator()
    try:
        op.set_device_output(device)
        op.add_input(omg.make_batch([L, L, D], [key, v, d], nulls))
        outs = op.drain()
    finally:
        op.delete()
        fac.close()
    held = memory()
    parts = [omg.batch_to_numpy(omg.batch_to_host(b) if device else b) for b in outs]
    omg.free_batches(outs)
    cols = [(np.concatenate([p[c][0] for p in parts]), np.concatenate([p[c][1] for p in parts])) for c in range(5)]
    order = np.argsort(cols[0][0])
    assert np.array_equal(cols[0][0][order], np.arange(100))
    assert np.array_equal(cols[1][0][order], np.bincount(key, weights=np.where(nulls[1], 0, v), minlength=100))
    assert np.array_equal(cols[2][0][order], np.bincount(key[~nulls[1]], minlength=100))
    assert np.array_equal(cols[3][1][order], np.arange(100) % 3 == 0)
    live = np.arange(100) % 3 != 0
    assert np.array_equal(cols[3][0][order][live], np.bincount(key, weights=d, minlength=100)[live])
    assert np.array_equal(cols[4][0][order], np.bincount(key, minlength=100))
    assert (held[0] if device else held[2]) - (before[0] if device else before[2]) <= 320 << 10
