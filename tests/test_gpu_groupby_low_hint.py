"""Group-bys whose hint is below the groups there are: what each partition's
table takes on chip is emitted from there, however many groups the table in
memory has slots for."""
import numpy as np
import pytest

from gpu_util import cpu_threads, dev, host, sort_groups
from proteus_gb300 import engine

pytestmark = pytest.mark.gpu


# 8 bits: partitions of 39,000, 65,536 and 23,000 rows; 9 bits and more: longer items
@pytest.mark.parametrize("n,hint,groups", [(10_000_000, 30_000, 90_000), (1 << 24, 100_000, 270_000),
                                           (6_000_000, 5000, 12_000), (9_000_000, 400_000, 1_000_000)])
@pytest.mark.parametrize("theta", [0.0, 1.0])
def test_more_groups_than_hinted(ctx, oracle, n, hint, groups, theta):
    k, v = engine.gen_groupby(11, n, groups, theta)
    res = ctx.groupby(dev(k), dev(v), groups, expected_groups=hint)
    ctx.sync()
    got = sort_groups(*[host(c) for c in res[:5]], host(res[5])[0])
    exp = oracle.groupby(k, v, threads=cpu_threads())
    assert all((a == b).all() for a, b in zip(got, exp)) and len(got[0]) == len(exp[0])


def test_pool_without_room_for_the_larger_table(ctx, oracle):
    """The table for groups beyond the hint is not what makes a call fail."""
    n, groups = 10_000_000, 5000
    k, v = engine.gen_groupby(12, n, groups, 1.0)
    d = dev(k), dev(v)
    ctx.sync()
    # pairs, the least table, offsets and items of 256 partitions, counters and cursors
    need = 8 * n + 28 * (1 << 14) + 16 * 257 + 8 * 512 + 4096
    ctx.set_pool_limit(ctx.pool_stats()["in_use"] + need)
    try:
        res = ctx.groupby(*d, groups, expected_groups=groups)
        ctx.sync()
    finally:
        ctx.set_pool_limit(0)
    got = sort_groups(*[host(c) for c in res[:5]], host(res[5])[0])
    assert all((a == b).all() for a, b in zip(got, oracle.groupby(k, v, threads=cpu_threads())))
