"""Aggregate lists of every length over both key widths, at probe counts around
a warp's 32 lanes and its match ring, with duplicate build keys, full buckets
and the lowest key (the side list), against the oracle."""
import numpy as np
import pytest

from gpu_util import dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu

LIST = [
    (abi.AGG_SUM, abi.VAL_BUILD), (abi.AGG_MIN, abi.VAL_PROBE), (abi.AGG_MAX, abi.VAL_PRODUCT),
    (abi.AGG_SUM, abi.VAL_BUILD_ROWID), (abi.AGG_MAX, abi.VAL_ROWID_XOR), (abi.AGG_MIN, abi.VAL_BUILD_KEY),
    (abi.AGG_AND, abi.VAL_BUILD), (abi.AGG_OR, abi.VAL_PROBE_ROWID),
]


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("unique", [False, True])
@pytest.mark.parametrize("n_probe,n_aggs", [(1, 1), (31, 2), (33, 4), (64, 5), (257, 8), (100_003, 3)])
def test_lists(ctx, oracle, dtype, unique, n_probe, n_aggs):
    rng = np.random.default_rng(n_probe)
    low = np.iinfo(dtype).min
    if unique:
        rk = rng.permutation(np.arange(-3000, 3000)).astype(dtype)
        rk[5] = low
    else:  # many copies of few keys: matches in several full buckets each
        rk = rng.integers(-40, 40, 3000).astype(dtype)
        rk[::500] = low
    rp = rng.integers(-1000, 1000, len(rk)).astype(np.int32)
    sk = rng.integers(-4000, 4000, n_probe).astype(dtype) if unique else rng.integers(-50, 50, n_probe).astype(dtype)
    sk[::29] = low
    sp = rng.integers(-1000, 1000, n_probe).astype(np.int32)
    aggs = LIST[:n_aggs]
    t = ctx.join_build(dev(rk), dev(rp))
    got = host(ctx.join_probe_agg(t, dev(sk), dev(sp), aggs)).tolist()
    ctx.sync()
    t.destroy()
    join = oracle.join_agg_i64 if dtype == np.int64 else oracle.join_agg
    assert got == join(rk, rp, sk, sp, aggs)


@pytest.mark.parametrize("n_build,copies", [(16, 1), (16, 16), (4000, 1), (8192, 1), (8192, 2), (8191, 5)])
def test_marked_buckets(ctx, oracle, n_build, copies):
    """int64 tables at load one half: rows that go past one and several full buckets are found, with the build rows
    of both slots of a marked bucket."""
    rng = np.random.default_rng(n_build + copies)
    rk = rng.permutation(np.arange(n_build) // copies).astype(np.int64) * 0x1_0000_0003
    rp = rng.integers(-1000, 1000, n_build).astype(np.int32)
    sk = rng.permutation(np.concatenate([rk[:3000], rk[:3000] + 1, rk[-3000:]]))
    sp = rng.integers(-1000, 1000, len(sk)).astype(np.int32)
    aggs = [(abi.AGG_COUNT, abi.VAL_ONE), (abi.AGG_SUM, abi.VAL_PRODUCT), (abi.AGG_SUM, abi.VAL_ROWID_XOR)]
    t = ctx.join_build(dev(rk), dev(rp))
    got = host(ctx.join_probe_agg(t, dev(sk), dev(sp), aggs)).tolist()
    ctx.sync()
    t.destroy()
    assert got == oracle.join_agg_i64(rk, rp, sk, sp, aggs)
