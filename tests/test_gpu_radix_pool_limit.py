"""An untuned radix join in the pool that the fewest partitions need: both sides
as pairs, and a few words for each partition."""
import numpy as np
import pytest

from gpu_util import CONFIG2_AGGS, cpu_threads, dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,ns", [(1, 3), (4000, 9000), (10_000, 20_000), (300_000, 600_000), (1_000_000, 2_000_000)])
def test_fewest_partitions(ctx, oracle, nr, ns):
    rng = np.random.default_rng(nr)
    rk = rng.permutation(nr).astype(np.int32) * 3
    sk = rng.integers(0, 2 * nr, ns).astype(np.int32) * 3
    d = dev(rk), None, dev(sk), None
    bits = 1
    while nr / 2**bits + 5 * (nr / 2**bits) ** 0.5 > 4608:
        bits += 1
    ctx.sync()
    # five tables of a partition's words (offsets of both sides, items, counts, cursors), each of some 256-byte units
    ctx.set_pool_limit(ctx.pool_stats()["in_use"] + 8 * (nr + ns) + 5 * 8 * 2**bits + 9 * 256)
    try:
        got = ctx.radix_join_agg(*d, CONFIG2_AGGS)
        ctx.sync()
    finally:
        ctx.set_pool_limit(0)
    assert host(got).tolist() == oracle.radix_join_agg(rk, None, sk, None, CONFIG2_AGGS, threads=cpu_threads())
