"""Grouping int64 keys with values where the pool has 40 bytes a slot and no
more: the table that keeps its counts in the records, through the on-chip level
and without it, against the oracle and at the number of groups it takes."""
import numpy as np
import pytest

from gpu_util import dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu
MIN = np.iinfo(np.int64).min


def limited(ctx, slots, call):
    ctx.sync()
    ctx.set_pool_limit(ctx.pool_stats()["in_use"] + 40 * (slots + 1) + 1024)
    try:
        got = call()
        ctx.sync()
        return got
    finally:
        ctx.set_pool_limit(0)


# slots: the power of two from twice the expected groups (1024 at least)
@pytest.mark.parametrize("n,groups,expected,slots", [(1, 1, 1, 2048), (70_001, 900, 900, 2048), (5000, 2048, 2048, 4096),
                                                     (300_001, 5000, 5000, 16384), (1 << 20, 200_000, 200_000, 1 << 19)])
@pytest.mark.parametrize("i64_values", [True, False])
def test_forty_bytes_a_slot(ctx, oracle, n, groups, expected, slots, i64_values):
    rng = np.random.default_rng(n)
    keys = rng.integers(-(1 << 62), 1 << 62, groups)[rng.integers(0, groups, n)]
    keys[::997] = MIN
    if i64_values:
        vals = rng.integers(-(1 << 63), (1 << 63) - 1, n)
        dk, dv = dev(keys), dev(vals)
        got = limited(ctx, slots, lambda: ctx.nest_i64(dk, dv, n + 1, expected_groups=expected))
    else:
        vals = rng.integers(-(1 << 31), (1 << 31) - 1, n)
        dk, dv = dev(keys), dev(vals.astype(np.int32))
        got = limited(ctx, slots, lambda: ctx.groupby(dk, dv, n + 1, expected_groups=expected))
    m = int(host(got[5])[0])
    order = np.argsort(host(got[0])[:m])
    for g, e in zip(got[:5], oracle.nest_i64(keys, vals)):
        assert (host(g)[:m][order] == e).all()


@pytest.mark.parametrize("extra", [0, 1])
def test_groups_it_takes(ctx, extra):
    keys = np.arange(8192 + extra, dtype=np.int64) * 3
    keys = np.concatenate([keys, keys, [MIN]]).astype(np.int64)
    d = dev(keys)
    if extra:
        with pytest.raises(abi.GbjError) as e:
            limited(ctx, 8192, lambda: ctx.nest_i64(d, d, 10_000, expected_groups=2500))
        assert e.value.code == abi.ERR_CAPACITY
    else:
        got = limited(ctx, 8192, lambda: ctx.nest_i64(d, d, 10_000, expected_groups=2500))
        assert int(host(got[5])[0]) == 8193
