"""Small aggregations (one launch, AUTO up to 16,384 rows in at most 8 steps of 2048) against the oracle."""
import numpy as np
import pytest

import omnioperator_gb300 as omg
from test_gpu_agg import _check_cfg1, _uniform_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,groups,batches", [(1, 1, (1,)), (2047, 40, (2047,)), (2048, 2000, (2048,)), (2049, 3, (2049,)),
                                              (16384, 900, (16384,)), (16385, 900, (16385,)), (8 * 700, 50, (700,)),
                                              (9 * 700, 50, (700,))])
def test_sizes_around_the_steps(gpu, n, groups, batches):
    """One row, a step and its neighbours, the largest call and the next, and as many ragged batches as steps
    (and one more); NULL values, NULL keys and the EMPTY key."""
    key, v1, v2, km, m1, m2 = _uniform_case(n, groups, n, nulls=0.05, key_nulls=0.03)
    key[n // 2::97] = np.iinfo(np.int64).min
    ctr = _check_cfg1(key, v1, v2, km, m1, m2, batch_sizes=batches)
    fits = n <= 16384 and len(range(0, n, batches[0])) <= 8
    assert (ctr["launches"] == 1) == fits


@pytest.mark.parametrize("device_input", [False, True])
def test_more_groups_than_the_table_holds(gpu, device_input):
    """The launch writes nothing and the regular path runs."""
    key, v1, v2, km, m1, m2 = _uniform_case(16_000, 10**6, 5)
    ctr = _check_cfg1(key, v1, v2, km, m1, m2, batch_sizes=(8000,), device_input=device_input)
    assert ctr["launches"] > 1
