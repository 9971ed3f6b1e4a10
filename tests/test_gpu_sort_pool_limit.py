"""A sort in the pool that it always had enough of: two words for each row
twice, and a 4-byte count and an 8-byte offset of each digit for every 2048 rows."""
import numpy as np
import pytest

from gpu_util import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8193, 10_000, 12_289, 65_537, 300_000, (1 << 20) - 1, 1 << 20, 3_000_001])
@pytest.mark.parametrize("n_cols", [1, 2, 3])
def test_bytes_a_row(ctx, n, n_cols):
    rng = np.random.default_rng(n)
    cols = [rng.integers(-(1 << 31), 1 << 31, n).astype(np.int32) for _ in range(n_cols)]
    d = [dev(c) for c in cols]
    ctx.sync()
    ctx.set_pool_limit(ctx.pool_stats()["in_use"] + 16 * n + 12 * 256 * -(-n // 2048) + 1024)
    try:
        out = ctx.sort_by_key(d, 0)
        ctx.sync()
    finally:
        ctx.set_pool_limit(0)
    order = np.argsort(cols[0], kind="stable")
    for o, c in zip(out, cols):
        assert (host(o) == c[order]).all()
