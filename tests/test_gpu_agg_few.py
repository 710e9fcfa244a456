"""Group-by with a handful of groups (thread-private states, chosen by AUTO) against the oracle: integers and
decimals bit-exact, double SUM/AVG within the stated tolerance."""
import numpy as np
import pytest

import omnioperator_gb300 as omg
import oracle
from helpers import assert_agg_equal, exact_by_key, run_agg
from test_gpu_agg import _check_cfg1, _uniform_case

pytestmark = pytest.mark.gpu

L, D, I = omg.LongType(), omg.DoubleType(), omg.IntType()
D64, D128 = omg.Decimal64Type(18, 2), omg.Decimal128Type(38, 2)
SUM, CALL, AVG = omg.OMNI_AGGREGATION_TYPE_SUM, omg.OMNI_AGGREGATION_TYPE_COUNT_ALL, omg.OMNI_AGGREGATION_TYPE_AVG


@pytest.mark.parametrize("n,groups,nulls,key_nulls", [(1 << 18, 1, 0.0, 0.0), (300_001, 2, 0.02, 0.0), (500_000, 9, 0.0, 0.01),
                                                      (700_000, 6, 0.02, 0.01), (400_003, 12, 0.0, 0.0)])
def test_few_groups(gpu, n, groups, nulls, key_nulls):
    """Around the groups that fit (11 of this plan without NULLs, fewer with them), with NULL and EMPTY keys
    and ragged batches."""
    key, v1, v2, km, m1, m2 = _uniform_case(n, groups, n + groups, nulls=nulls, key_nulls=key_nulls)
    key[7::5000] = np.iinfo(np.int64).min
    _check_cfg1(key, v1, v2, km, m1, m2, batch_sizes=(4096, 1000, 777))


def test_more_groups_than_estimated(gpu):
    """The hint says 3 groups: those beyond the private ones go to the global table row by row."""
    key, v1, v2, km, m1, m2 = _uniform_case(300_000, 60, 11)
    ctr = _check_cfg1(key, v1, v2, km, m1, m2, strategy=omg.AGG_STRATEGY_AUTO, capacity_hint=3,
                      batch_sizes=(300_000,))
    assert ctr["sizing"]["estimate"] == 3


def test_packed_keys_exact_sums(gpu):
    """NULLs inside a packed key; decimal sums of magnitudes on both sides of 2^57 and of both signs."""
    rng = np.random.default_rng(12)
    n = 600_000
    k1 = rng.integers(0, 2, n).astype(np.int32)
    k2 = rng.integers(0, 2, n).astype(np.int64) << 40
    km = rng.random(n) < 0.1
    dec = rng.integers(-10**17, 10**17, n, dtype=np.int64)
    dec[::3] = rng.integers(-10**18 + 1, 10**18, len(dec[::3]), dtype=np.int64)
    dec[1::3] = rng.integers(-50, 50, len(dec[1::3]))
    dm = rng.random(n) < 0.02
    v = rng.standard_normal(n)
    vm = rng.random(n) < 0.02
    cols, ctr = run_agg([0, 1], [I, L], [[2], [], [3]], [[D64], [], [D]], [[D128], [L], [D]], [SUM, CALL, AVG],
                        [k1, k2, dec, v], [I, L, D64, D], nulls=[km, None, dm, vm], batch_sizes=(65536, 333))
    assert ctr["sizing"]["part_bits"] == 0
    ora = oracle.hashagg([k1, k2], [oracle.T_INT, oracle.T_LONG], [km, None],
                         [dict(func=oracle.F_SUM, col=dec, in_type=oracle.T_DEC64, out_type=oracle.T_DEC128, nulls=dm),
                          dict(func=oracle.F_COUNT_ALL, col=None, out_type=oracle.T_LONG),
                          dict(func=oracle.F_AVG, col=v, in_type=oracle.T_DOUBLE, out_type=oracle.T_DOUBLE, nulls=vm)])
    ex = exact_by_key([k1, k2], [km, None], v, ~vm, divide_by_count=True)
    assert_agg_equal(cols, ora, 2, double_aggs=(2,), exact={2: ex})
