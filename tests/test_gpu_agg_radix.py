"""Radix aggregation (more groups than the partitioned strategy holds, chosen by AUTO from the key
sketch) against the oracle: integers bit-exact, double SUM/AVG within the stated tolerance."""
import numpy as np
import pytest

import omnioperator_gb300 as omg
import oracle
from helpers import assert_agg_equal, exact_by_key, run_agg
from test_gpu_agg import _cfg1_aggs, _check_cfg1, _uniform_case

pytestmark = pytest.mark.gpu

L, D, I = omg.LongType(), omg.DoubleType(), omg.IntType()
D64, D128 = omg.Decimal64Type(18, 2), omg.Decimal128Type(38, 2)
SUM, CNT, CALL, AVG = (omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_COLUMN,
                       omg.OMNI_AGGREGATION_TYPE_COUNT_ALL, omg.OMNI_AGGREGATION_TYPE_AVG)
MIN, MAX = omg.OMNI_AGGREGATION_TYPE_MIN, omg.OMNI_AGGREGATION_TYPE_MAX


def _radix(ctr):
    """The run's sizing record says AUTO left the partitioned strategy."""
    return ctr["sizing"]["part_bits"] == -1 and ctr["sizing"]["rows"] >= 1 << 18


@pytest.mark.parametrize("n,groups,batches", [(1 << 19, 2_000_000, (4096, 1000, 777)), (600_001, 350_000, (600_001,)),
                                              (600_000, 600_000, (65536, 13))])
def test_many_groups_with_nulls(gpu, n, groups, batches):
    """Ragged tiles, NULL values, NULL keys and the EMPTY key (the special groups)."""
    key, v1, v2, km, m1, m2 = _uniform_case(n, groups, n, nulls=0.02, key_nulls=0.01)
    key[5::1000] = np.iinfo(np.int64).min
    ctr = _check_cfg1(key, v1, v2, km, m1, m2, batch_sizes=batches)
    assert _radix(ctr)


@pytest.mark.parametrize("share,nulls", [(0.3, 0.0), (0.55, 0.02)])
def test_hot_keys_are_split_over_units(gpu, share, nulls):
    """Two keys hold `share` of the rows: their partitions are cut into units of 2^14 rows whose
    tables meet in the global table, the hottest group of a unit on its replicas."""
    key, v1, v2, km, m1, m2 = _uniform_case(1_500_000, 1_200_000 if share < 0.5 else 130_000, 3, nulls=nulls)
    rng = np.random.default_rng(4)
    u = rng.random(len(key))
    if share > 0.5:
        cold = u >= share
        key[cold] = rng.integers(-2**62, 2**62, int(cold.sum()), dtype=np.int64)
    key[u < share] = 77
    key[u < share / 4] = -12345
    ctr = _check_cfg1(key, v1, v2, km, m1, m2, batch_sizes=(500_000,))
    assert _radix(ctr)


def test_packed_keys_decimal_sum_and_avg(gpu):
    """A record with 4-, 8- and 16-byte values and NULL bytes: (INT, DECIMAL128) keys."""
    rng = np.random.default_rng(5)
    n = 500_000
    code = rng.integers(0, 300_000, n)
    k1 = (code % 65521).astype(np.int32)
    k2 = np.stack([code.astype(np.uint64) * 2654435761, np.zeros(n, np.uint64)], axis=1)
    km = code % 113 == 7
    dec = rng.integers(-10**9, 10**9, n, dtype=np.int64)
    dm = rng.random(n) < 0.02
    v = rng.standard_normal(n)
    vm = rng.random(n) < 0.02
    cols, ctr = run_agg([0, 1], [I, D128], [[2], [], [3]], [[D64], [], [D]], [[D128], [L], [D]],
                        [SUM, CALL, AVG], [k1, k2, dec, v], [I, D128, D64, D], nulls=[km, None, dm, vm],
                        batch_sizes=(65536, 999))
    assert _radix(ctr)
    # The oracle groups by the low word of the second key (the high word is 0).
    got = [cols[0], (cols[1][0][:, 0].astype(np.int64), cols[1][1])] + cols[2:]
    assert not cols[1][0][:, 1].any()
    k2 = k2[:, 0].astype(np.int64)
    ora = oracle.hashagg([k1, k2], [oracle.T_INT, oracle.T_LONG], [km, None],
                         [dict(func=oracle.F_SUM, col=dec, in_type=oracle.T_DEC64, out_type=oracle.T_DEC128, nulls=dm),
                          dict(func=oracle.F_COUNT_ALL, col=None, out_type=oracle.T_LONG),
                          dict(func=oracle.F_AVG, col=v, in_type=oracle.T_DOUBLE, out_type=oracle.T_DOUBLE, nulls=vm)])
    ex = exact_by_key([k1, k2], [km, None], v, ~vm, divide_by_count=True)
    assert_agg_equal(got, ora, 2, double_aggs=(2,), exact={2: ex})


def test_second_flush_after_a_radix_flush(gpu):
    """The first flush's groups move from the dense array into the table for the rows that follow."""
    key, v1, v2, km, m1, m2 = _uniform_case(1_100_000, 1_500_000, 6, key_nulls=0.01)
    omg.lib().omg_debug_set_agg_flush_rows(500_000)
    try:
        ctr = _check_cfg1(key, v1, v2, km, m1, m2, batch_sizes=(100_000,))
    finally:
        omg.lib().omg_debug_set_agg_flush_rows(0)
    assert _radix(ctr)


def test_order_dependent_overflow_after_a_radix_run(gpu):
    """A decimal128 SUM that leaves the bound on a row-ordered prefix and comes back: the replay
    finds its group although the groups were dense."""
    n = 400_000
    key = np.random.default_rng(7).integers(0, 250_000, n).astype(np.int64)
    vals = np.zeros((n, 2), np.uint64)
    vals[:, 0] = np.arange(n)
    big = 10**38 - 1
    for r, x in zip(np.nonzero(key == key[100])[0][:1].tolist() + [n - 3, n - 2], (big, big, -big)):
        key[r] = key[100]
        vals[r] = [x & (2**64 - 1), (x >> 64) & (2**64 - 1)]
    d = omg.Decimal128Type(38, 0)
    cols, ctr = run_agg([0], [L], [[1]], [[d]], [[d]], [SUM], [key, vals], [L, d], overflow_as_null=True,
                        batch_sizes=(100_000,))
    assert _radix(ctr) and ctr["ordered_groups"] >= 1
    ora = oracle.hashagg([key], [oracle.T_LONG], [None],
                         [dict(func=oracle.F_SUM, col=vals, in_type=oracle.T_DEC128, out_type=oracle.T_DEC128)],
                         overflow_as_null=True)
    assert_agg_equal(cols, ora, 1)


def test_several_passes_over_a_partition(gpu):
    """More groups than 2^14 partitions of a wide plan's shared tables hold (five decimal128 sums, over 350
    bytes a group): a partition takes several passes.  Every key is unique, so the sums are the inputs."""
    n = 4_000_000
    key = np.random.default_rng(8).permutation(n).astype(np.int64) * 7919
    vals = np.zeros((n, 2), np.uint64)
    vals[:, 0] = np.arange(n, dtype=np.uint64) + 1
    cols, ctr = run_agg([0], [L], [[c] for c in range(1, 6)], [[D128]] * 5, [[D128]] * 5, [SUM] * 5,
                        [key] + [vals] * 5, [L] + [D128] * 5, batch_sizes=(n,))
    order = np.argsort(cols[0][0], kind="stable")
    want = np.argsort(key, kind="stable")
    assert np.array_equal(cols[0][0][order], key[want])
    for v, m in cols[1:]:
        assert not m.any() and np.array_equal(v[order], vals[want])
