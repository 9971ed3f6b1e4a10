"""Group-by work items on the GPU vs the oracle: their edges, and partitions of several items."""
import numpy as np
import pytest

from test_gpu_groupby import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 8191, 8192, 8193, 32767, 32769, 65537, 3 * 32768 + 1, 2_000_003])
@pytest.mark.parametrize("strategy", [1, 2])
@pytest.mark.parametrize("hot", [0.0, 0.9])
def test_item_edges(ctx, oracle, rows, strategy, hot):
    """`hot`: the share of the rows that one key takes, so that its partition spans items and the last one is short."""
    rng = np.random.default_rng(rows)
    k = rng.integers(-4000, 4000, rows, dtype=np.int32)
    k[rng.random(rows) < hot] = np.iinfo(np.int32).min if rows % 2 else 17
    v = rng.integers(-(1 << 31), 1 << 31, rows, dtype=np.int64).astype(np.int32)
    check(ctx, oracle, k, v, expected_groups=8001, strategy=strategy)


@pytest.mark.parametrize("groups", [1 << 9, 1 << 17, 1 << 18, 1 << 20])
def test_partition_counts(ctx, oracle, groups):
    """One narrow pass, one wide pass, and two passes' worth of bits; every sixth row has the same key."""
    rows = 3_000_001
    rng = np.random.default_rng(groups)
    k = rng.integers(0, groups, rows, dtype=np.int64).astype(np.int32) * 7 - (1 << 20)
    k[::6] = k[0]
    v = rng.integers(-1000, 1000, rows, dtype=np.int32)
    check(ctx, oracle, k, v, expected_groups=groups, strategy=2)


@pytest.mark.parametrize("groups", [1, 16, 300, 5000])
def test_sum_carries(ctx, oracle, groups):
    """Sums whose low 32 bits carry at every row, at none, and once in 2^16 rows; more rows a group than a flush holds."""
    rows = 400_001
    k = (np.arange(rows) % groups).astype(np.int32)
    for v in (np.full(rows, np.iinfo(np.int32).max, np.int32), np.full(rows, np.iinfo(np.int32).min, np.int32),
              np.full(rows, -(1 << 31) + (1 << 16), np.int64).astype(np.int32)):
        check(ctx, oracle, k, v, expected_groups=groups)
