"""Group-bys on 9 and 11 bits (one wide pass) and on 13 and 14 (two passes), with
a partition of several items."""
import numpy as np
import pytest

from test_gpu_groupby import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,rows", [(1 << 19, 4_000_000), (1 << 21, 6_000_000), (5_000_000, 6_000_000),
                                         (9_000_000, 9_500_000)])
def test_bits(ctx, oracle, groups, rows):
    rng = np.random.default_rng(groups)
    k = rng.permutation(rows).astype(np.int32) % np.int32(groups) - np.int32(1 << 20)
    k[::6] = k[0]
    v = rng.integers(-1000, 1000, rows, dtype=np.int32)
    check(ctx, oracle, k, v, expected_groups=groups, strategy=2)
