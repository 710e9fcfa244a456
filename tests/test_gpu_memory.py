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
