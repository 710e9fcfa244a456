"""Batched aggregation (many tasks, one persistent launch, CUDA graph, autotuned shape) against
the oracle task by task: every task's output must equal a separate HashAggregation of that task
(bit-exact integers, doubles within the stated tolerance), including tasks re-run through the
exact path when their table overflows."""
import numpy as np
import pytest

import omnioperator_gb300 as omg
import omnioperator_gb300.sizer as sz
from helpers import assert_agg_equal, exact_by_key
from test_gpu_agg import _cfg1_aggs, _cfg1_oracle

pytestmark = pytest.mark.gpu

L, D = omg.LongType(), omg.DoubleType()


def _tasks(seed, n_tasks, max_rows=60_000, nulls=False):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n_tasks):
        n = int(np.exp(rng.uniform(0, np.log(max_rows))))
        d = int(np.exp(rng.uniform(np.log(2), np.log(max(3, n)))))
        uniq = rng.integers(-2**62, 2**62, d, dtype=np.int64)
        key = uniq[rng.integers(0, d, n)]
        v1 = rng.integers(-10**6, 10**6, n, dtype=np.int64)
        v2 = rng.random(n)
        km = rng.random(n) < 0.02 if nulls else None
        m1 = rng.random(n) < 0.05 if nulls else None
        m2 = rng.random(n) < 0.05 if nulls else None
        out.append((key, v1, v2, km, m1, m2))
    return out


def _run(tasks, flags=0, sizer=None, runs=1):
    fac = omg.HashAggregationOperatorFactory(**{k: v for k, v in zip(
        ["group_by_cols", "group_input_types", "aggs_cols", "agg_input_types", "agg_output_types", "agg_func_types"],
        _cfg1_aggs().values())})
    handles = [omg.make_batch([L, L, D], [k, a, b], [km, m1, m2]) for k, a, b, km, m1, m2 in tasks]
    batch = omg.AggBatch(fac, handles, sizer=sizer, flags=flags)
    results = []
    for _ in range(runs):
        batch.run()
        per = {}
        for t, b in batch.outputs():
            if flags & omg.BATCH_DEVICE_OUTPUT:
                h = omg.batch_to_host(b)
                omg.free_batch(b)
                b = h
            per.setdefault(t, []).append(omg.batch_to_numpy(b))
            omg.free_batch(b)
        results.append(per)
    info = batch.info()
    batch.close()
    omg.free_batches(handles)
    fac.close()
    return results, info


def _check(tasks, per):
    for t, (key, v1, v2, km, m1, m2) in enumerate(tasks):
        parts = per.get(t, [])
        cols = [(np.concatenate([p[c][0] for p in parts]), np.concatenate([p[c][1] for p in parts]))
                for c in range(7)] if parts else None
        ora = _cfg1_oracle(key, km, v1, m1, v2, m2)
        valid = None if m2 is None else ~m2
        ex_sum = exact_by_key([key], [km], v2, valid)
        ex_avg = exact_by_key([key], [km], v2, valid, divide_by_count=True)
        assert_agg_equal(cols, ora, 1, double_aggs=(4, 5), exact={4: ex_sum, 5: ex_avg})


def test_batched_equals_separate_aggregations(gpu):
    tasks = _tasks(1, 120, nulls=True)
    (per,), info = _run(tasks)
    _check(tasks, per)
    # plain sizing may undersize a few tables; those tasks take the exact re-run path
    assert info["tasks"] == 120 and info["graph"] == 1 and info["reruns"] <= 12
    assert info["threads"] in (128, 256, 512, 1024)


def test_batched_graph_replays_give_the_same_result(gpu):
    tasks = _tasks(2, 60)
    (first, second), info = _run(tasks, runs=2)
    _check(tasks, first)
    _check(tasks, second)
    assert info["runs"] == 2 and info["graph"] == 1


def test_batched_overflowing_tasks_rerun_exactly(gpu):
    tasks = _tasks(3, 40, max_rows=20_000, nulls=True)
    (per,), info = _run(tasks, flags=omg.BATCH_DEBUG_TINY_TABLES)
    _check(tasks, per)
    assert info["reruns"] >= 5


@pytest.mark.parametrize("flags", [0, omg.BATCH_DEVICE_OUTPUT | omg.BATCH_NO_GRAPH])
def test_batched_grow_pass_finishes_overflowing_tasks(gpu, flags):
    """64-slot first tables: the tasks that outgrow them take one more batched run with tables of
    twice their rows (no operator re-runs), equal to the oracle task by task, over graph replays."""
    tasks = _tasks(5, 40, max_rows=20_000, nulls=True)
    (first, second), info = _run(tasks, flags=flags | omg.BATCH_DEBUG_TINY_GROW, runs=2)
    _check(tasks, first)
    _check(tasks, second)
    assert info["reruns"] >= 5 and info["grown"] == info["reruns"] and info["operator_reruns"] == 0


def test_batched_device_output_without_graph(gpu):
    tasks = _tasks(4, 50)
    (per,), info = _run(tasks, flags=omg.BATCH_DEVICE_OUTPUT | omg.BATCH_NO_GRAPH | omg.BATCH_NO_TUNE)
    _check(tasks, per)
    assert info["graph"] == 0


def test_batched_with_learned_sizer(gpu):
    model = sz.SizingModel.load(str(__import__("pathlib").Path(omg.__file__).parent / "models" / "agg_sizer.json"))
    tasks = _tasks(5, 80)
    (per,), info = _run(tasks, sizer=model)
    _check(tasks, per)
    assert info["learned"] == 1
    model.close()


@pytest.mark.parametrize("groups", [1, 511, 512, 1023, 1024, 1025, 9000])
def test_batched_tables_around_a_chunk_of_slots(gpu, groups):
    """Tables are counted and extracted 2048 slots at a time: group counts whose tables end just
    below, at and just past a chunk (two special slots follow the power-of-two capacity), next to a
    one-row task and NULL and EMPTY keys (the special slots of the last chunk)."""
    rng = np.random.default_rng(groups)
    tasks = []
    for n in (1, 3 * groups + 7):
        key = (np.arange(n) % groups).astype(np.int64) * 7919
        key[-1] = np.iinfo(np.int64).min
        km = np.arange(n) % 97 == 5
        tasks.append((key, rng.integers(-10**6, 10**6, n, dtype=np.int64), rng.random(n), km, None, None))
    (per,), _ = _run(tasks)
    _check(tasks, per)


@pytest.mark.parametrize("groups", [255, 300, 1100, 2300, 9000, 11_000, 40_000])
def test_batched_units_and_partitions(gpu, groups):
    """Tasks whose rows go through shared tables, by units of 8 tiles and more, in one to eight partitions, and
    just past those: rows around a unit's end, NULL and EMPTY keys, NULL values, double sums."""
    rng = np.random.default_rng(groups)
    tasks = []
    for n in (32_768, 32_769, 140_001):
        key = rng.integers(0, groups, n) * 7919
        key[::1009] = np.iinfo(np.int64).min
        tasks.append((key, rng.integers(-2**40, 2**40, n, dtype=np.int64), rng.random(n), rng.random(n) < 0.02,
                      rng.random(n) < 0.05, rng.random(n) < 0.05))
    (per, again), _ = _run(tasks, runs=2)
    _check(tasks, per)
    _check(tasks, again)


@pytest.mark.parametrize("groups", [1, 7, 3000])
def test_batched_units_of_two_column_keys(gpu, groups):
    """Whole-number states of few groups and a packed key in the units' shared tables, exact in numpy."""
    rng = np.random.default_rng(groups)
    I = omg.IntType()
    fac = omg.HashAggregationOperatorFactory([0, 1], [I, L], [[2], [2]], [[L], [L]], [[L], [L]],
                                             [omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_COLUMN])
    data = []
    for n in (1, 4097, 70_001):
        code = rng.integers(0, groups, n)
        data.append((code.astype(np.int32) % 13, code * 2**33, rng.integers(-2**45, 2**45, n), rng.random(n) < 0.1))
    handles = [omg.make_batch([I, L, L], [a, b, v], [None, None, m]) for a, b, v, m in data]
    batch = omg.AggBatch(fac, handles)
    batch.run()
    got = {}
    for t, b in batch.outputs():
        got.setdefault(t, []).append(omg.batch_to_numpy(b))
        omg.free_batch(b)
    batch.close()
    omg.free_batches(handles)
    fac.close()
    for t, (a, b, v, m) in enumerate(data):
        cols = [np.concatenate([p[c][0] for p in got[t]]) for c in range(4)]
        null = np.concatenate([p[2][1] for p in got[t]])
        code, inv = np.unique(b // 2**33, return_inverse=True)
        order = np.argsort(cols[1])
        assert np.array_equal(cols[1][order], code * 2**33)
        assert np.array_equal(cols[0][order], code % 13)
        want = np.zeros(len(code), np.int64)
        np.add.at(want, inv[~m], v[~m])
        count = np.bincount(inv[~m], minlength=len(code))
        assert np.array_equal(~null[order], count > 0)
        assert np.array_equal(cols[2][order][count > 0], want[count > 0])
        assert np.array_equal(cols[3][order], count)


def test_tuning_times_the_tasks_that_the_launch_is_for(gpu):
    """Tasks that go by units leave the launch nothing to time, and what was found for one number of rows in the tasks'
    own tables is not taken for another."""
    rng = np.random.default_rng(41)
    # Seven sums of one column of its own each: a plan shape that no other test tunes.
    fac = omg.HashAggregationOperatorFactory([0], [L], [[c] for c in range(1, 8)], [[L]] * 7, [[L]] * 7,
                                             [omg.OMNI_AGGREGATION_TYPE_SUM] * 7)

    def tuned(groups):
        tasks = []
        for g in groups:
            key = rng.integers(0, g, 60_000)
            tasks.append(omg.make_batch([L] * 8, [key] + [key * k for k in range(1, 8)]))
        batch = omg.AggBatch(fac, tasks)
        batch.run()
        for t, b in batch.outputs():
            cols = omg.batch_to_numpy(b)
            omg.free_batch(b)
            n = cols[1][0] // np.where(cols[0][0] == 0, 1, cols[0][0])  # rows of the group
            assert np.array_equal(cols[7][0], 7 * n * cols[0][0])
        us = batch.info()["tune_us"]
        batch.close()
        omg.free_batches(tasks)
        return us

    assert tuned([10] * 16) == 0
    assert tuned([50_000] * 16) > 0
    assert tuned([50_000] + [10] * 15) > 0
    assert tuned([50_000] * 15 + [10]) == 0  # as sixteen, to a power of two
    fac.close()
