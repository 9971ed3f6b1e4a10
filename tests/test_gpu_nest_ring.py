"""Grouping int64 keys in the global table: row counts around a warp and its
ring, groups whose home slots collide, INT64_MIN, every value form, and the
number of groups a table takes, against the oracle."""
import numpy as np
import pytest

from gpu_util import dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_vals", [True, False])
@pytest.mark.parametrize("n,groups,expected", [(1, 1, 0), (33, 20, 4000), (65, 65, 0), (4097, 4000, 4000),
                                               (100_003, 60_000, 60_000), (300_001, 3000, 2500),
                                               (200_000, 7, 70_000)])
def test_global_table(ctx, oracle, n, groups, expected, with_vals):
    rng = np.random.default_rng(n)
    keys = rng.integers(-(1 << 62), 1 << 62, groups)[rng.integers(0, groups, n)]
    keys[::97] = np.iinfo(np.int64).min
    vals = rng.integers(-(1 << 63), (1 << 63) - 1, n) if with_vals else None
    got = ctx.nest_i64(dev(keys), dev(vals) if with_vals else None, n + 1, expected_groups=expected)
    ctx.sync()
    m = int(host(got[5])[0])
    order = np.argsort(host(got[0])[:m])
    for g, e in zip(got[:5], oracle.nest_i64(keys, vals)):
        assert (host(g)[:m][order] == e).all()


@pytest.mark.parametrize("extra,ok", [(0, True), (1, False)])
@pytest.mark.parametrize("with_min", [False, True])
def test_groups_a_table_takes(ctx, extra, ok, with_min):
    """expected_groups = 2500 sizes it for 8192 groups, whatever its slots."""
    keys = np.arange(8192 + extra, dtype=np.int64) * 3
    keys = np.concatenate([keys, keys, [np.iinfo(np.int64).min] * with_min]).astype(np.int64)
    got = ctx.nest_i64(dev(keys), dev(keys), 10_000, expected_groups=2500)
    if ok:
        ctx.sync()
        assert int(host(got[5])[0]) == 8192 + with_min
    else:
        with pytest.raises(abi.GbjError) as e:
            ctx.sync()
        assert e.value.code == abi.ERR_CAPACITY


def test_long_chains(ctx, oracle):
    """Keys of one home slot: every row is looked up again and again, so that
    the warps' rings are full while new rows arrive."""
    rng = np.random.default_rng(9)
    cand = rng.integers(-(1 << 62), 1 << 62, 1 << 21)
    h = cand.astype(np.uint64)
    for factor in (0xFF51AFD7ED558CCD, 0xC4CEB9FE1A85EC53):  # the table's placement hash
        h ^= h >> np.uint64(33)
        h *= np.uint64(factor)
    h ^= h >> np.uint64(33)
    chain = cand[(h & np.uint64(32767)) == 0]
    assert len(chain) > 40
    keys = chain[rng.integers(0, len(chain), 2_000_000)]  # several rounds of every warp
    vals = rng.integers(-1000, 1000, len(keys))
    got = ctx.nest_i64(dev(keys), dev(vals), 1000, expected_groups=2500)
    ctx.sync()
    m = int(host(got[5])[0])
    order = np.argsort(host(got[0])[:m])
    for g, e in zip(got[:5], oracle.nest_i64(keys, vals)):
        assert (host(g)[:m][order] == e).all()


def test_table_at_the_pool_limit(ctx, oracle):
    """Where the pool has no room for a table of four times the slots, one of the least size is taken."""
    rng = np.random.default_rng(3)
    keys = rng.integers(0, 1 << 40, 4096)[rng.integers(0, 4096, 1 << 19)]
    vals = rng.integers(-1000, 1000, 1 << 19)
    dk, dv = dev(keys), dev(vals)
    ctx.sync()
    # 8192 slots (two for each group) of 48 bytes and the one of INT64_MIN; 32,768 would be 1.5 MB
    ctx.set_pool_limit(ctx.pool_stats()["in_use"] + 48 * 8193 + (1 << 16))
    try:
        got = ctx.nest_i64(dk, dv, 5000, expected_groups=4096)
        ctx.sync()
    finally:
        ctx.set_pool_limit(0)
    m = int(host(got[5])[0])
    order = np.argsort(host(got[0])[:m])
    for g, e in zip(got[:5], oracle.nest_i64(keys, vals)):
        assert (host(g)[:m][order] == e).all()
