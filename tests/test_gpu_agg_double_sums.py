"""SUM of doubles where the order and the splitting of the additions must not show: every path carries the
rounding errors of its additions along, so a sum is off by its own rounding and second-order terms only.

With u = 2^-53 and n rows, the carried errors are at most n u sum|x| and adding those up loses at most
n^2 u^2 sum|x|; turning sum and errors into the result rounds once more: u |sum|."""
import math

import numpy as np
import pytest

import omnioperator_gb300 as omg
from helpers import run_agg

pytestmark = pytest.mark.gpu

L, I, D = omg.LongType(), omg.IntType(), omg.DoubleType()
SUM, CALL = omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_ALL
U = 2.0**-53


def _values(kind, n, rng):
    if kind == "constant":
        return np.full(n, 0.1)
    if kind == "thirds":
        return rng.choice([0.1, 0.3, 1 / 3], n)
    big = np.tile([1e16, 1.0, -1e16, 3.0], n // 4 + 1)[:n]  # cancels, but for the small ones
    return big


def _check(group, x, got):
    """got: {group: sum}, for the groups to look at."""
    for g, s in got.items():
        v = x[group == g]
        exact, n = math.fsum(v), len(v)
        assert abs(s - exact) <= U * abs(exact) + n * n * U * U * np.abs(v).sum(), (g, n, s, exact)


def _run(key, x, **kw):
    cols, ctr = run_agg([0], [L], [[1], []], [[D], []], [[D], [L]], [SUM, CALL], [key, x], [L, D], **kw)
    return dict(zip(cols[0][0].tolist(), cols[1][0].tolist())), ctr


@pytest.mark.parametrize("kind", ["constant", "thirds", "cancel"])
@pytest.mark.parametrize("n,groups", [(1 << 18, 1), (1 << 18, 5), (1_000_003, 3)])
def test_few_groups(gpu, kind, n, groups):
    """Thread-private states."""
    rng = np.random.default_rng(groups)
    key = rng.integers(0, groups, n)
    x = _values(kind, n, rng)
    got, ctr = _run(key, x, batch_sizes=(n,))
    assert ctr["sizing"]["part_bits"] == 0
    _check(key, x, got)


@pytest.mark.parametrize("kind", ["constant", "thirds", "cancel"])
@pytest.mark.parametrize("n,groups", [(2048, 1), (16_384, 1), (16_384, 3), (16_001, 40)])
def test_small_calls(gpu, kind, n, groups):
    """One launch for the whole call: rows sorted by group, runs of a thread's and a warp's rows."""
    rng = np.random.default_rng(n + groups)
    key = rng.integers(0, groups, n)
    x = _values(kind, n, rng)
    got, ctr = _run(key, x, batch_sizes=(n,))
    assert ctr["launches"] == 1
    _check(key, x, got)


@pytest.mark.parametrize("kind", ["constant", "thirds", "cancel"])
def test_radix_passes(gpu, kind):
    """A hot group, whose partition is cut into units; groups of some hundred and of a few rows."""
    n = 1 << 20
    rng = np.random.default_rng(2)
    key = 1000 + rng.integers(0, 400_000, n)
    u = rng.random(n)
    key[u < 0.5] = rng.integers(100, 600, int((u < 0.5).sum()))
    key[u < 0.2] = 7
    x = _values(kind, n, rng)
    got, ctr = _run(key, x, batch_sizes=(n,))
    _check(key, x, {g: s for g, s in got.items() if g < 600 or g % 4001 == 0})


@pytest.mark.parametrize("kind", ["constant", "thirds", "cancel"])
def test_batched_tasks_by_units(gpu, kind):
    """A task whose rows many CTAs add up in shared tables of their own."""
    n, groups = 400_000, 300
    rng = np.random.default_rng(3)
    key = rng.integers(0, groups, n)
    x = _values(kind, n, rng)
    fac = omg.HashAggregationOperatorFactory([0], [L], [[1], []], [[D], []], [[D], [L]], [SUM, CALL])
    task = omg.make_batch([L, D], [key, x])
    batch = omg.AggBatch(fac, [task])
    batch.run()
    got = {}
    for _, b in batch.outputs():
        cols = omg.batch_to_numpy(b)
        omg.free_batch(b)
        got.update(zip(cols[0][0].tolist(), cols[1][0].tolist()))
    assert batch.info()["reruns"] == 0 and len(got) == groups
    batch.close()
    omg.free_batch(task)
    fac.close()
    _check(key, x, got)
