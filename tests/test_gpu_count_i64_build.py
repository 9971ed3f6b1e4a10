"""The int64 match count's table: unique keys, copies, one key for all rows, the
lowest key, against numpy, at row counts around a warp and a block."""
import numpy as np
import pytest

from gpu_util import dev, host

pytestmark = pytest.mark.gpu
MIN = np.iinfo(np.int64).min


def count(r, s):
    rk, rc = np.unique(r, return_counts=True)
    at = np.searchsorted(rk, s).clip(max=len(rk) - 1)
    return int(rc[at][rk[at] == s].sum())


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 70_001, 1 << 18])
@pytest.mark.parametrize("copies", [1, 3, 1000])
def test_match_count(ctx, n, copies):
    rng = np.random.default_rng(n + copies)
    keys = rng.integers(-(1 << 62), 1 << 62, -(-n // copies))
    r = rng.permutation(np.resize(keys, n))
    r[::11] = MIN
    s = np.concatenate([rng.choice(keys, 2 * n), rng.integers(-(1 << 62), 1 << 62, n), [MIN] * 5])
    got = ctx.radix_join_count_i64(dev(r), dev(s))
    ctx.sync()
    assert int(host(got)[0]) == count(r, s)

