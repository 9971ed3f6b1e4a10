"""Select, bloom probe, gather, reduce and pair output at the sizes where their
tiles, look-back windows and buffers end, on aligned and unaligned columns,
against numpy and the oracle."""
import numpy as np
import pytest

from gpu_util import dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 8191, 8192, 8193, 33 * 8192, 200 * 8192 + 5]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("lo,hi", [(0, 99), (-5, 2000), (5000, 6000), (999, 999)])
def test_select(ctx, n, shift, lo, hi):
    col = np.random.default_rng(n).integers(0, 1000, n + shift).astype(np.int32)
    rows, cnt = ctx.select_range(dev(col)[shift:], lo, hi)
    ctx.sync()
    exp = np.nonzero((col[shift:] >= lo) & (col[shift:] <= hi))[0]
    assert int(host(cnt)[0]) == len(exp)
    assert (host(rows)[:len(exp)] == exp).all()


@pytest.mark.parametrize("n", SIZES)
def test_bloom(ctx, oracle, n):
    rng = np.random.default_rng(n)
    build, probe = rng.integers(0, 1 << 20, 3000).astype(np.int32), rng.integers(-(1 << 20), 1 << 20, n).astype(np.int32)
    f = ctx.bloom_build(dev(build), 1 << 14)
    rows, cnt = ctx.bloom_probe(f, dev(probe))
    ctx.sync()
    exp = np.nonzero(np.isin(probe & ((1 << 14) - 1), build & ((1 << 14) - 1)))[0]
    assert int(host(cnt)[0]) == len(exp) and (host(rows)[:len(exp)] == exp).all()
    ctx.bloom_destroy(f)


@pytest.mark.parametrize("n", [1, 511, 4 * 512 + 1, 1_000_003])
@pytest.mark.parametrize("n_aggs", [1, 2, 3, 8])
def test_gather_and_reduce(ctx, oracle, n, n_aggs):
    rng = np.random.default_rng(n)
    col, rows = rng.integers(-1000, 1000, 70_001).astype(np.int32), rng.integers(0, 70_001, n).astype(np.int32)
    assert (host(ctx.gather(dev(col), dev(rows))) == col[rows]).all()
    aggs = [(abi.AGG_SUM, abi.VAL_BUILD), (abi.AGG_MAX, abi.VAL_PRODUCT), (abi.AGG_MIN, abi.VAL_PROBE),
            (abi.AGG_COUNT, abi.VAL_ONE), (abi.AGG_SUM, abi.VAL_PROBE_ROWID), (abi.AGG_OR, abi.VAL_BUILD),
            (abi.AGG_AND, abi.VAL_BUILD), (abi.AGG_MIN, abi.VAL_BUILD_KEY)][:n_aggs]
    for r in (rows, None):
        got = host(ctx.reduce(dev(col), aggs, rows=None if r is None else dev(r))).tolist()
        assert got == oracle.reduce(col, aggs, rows=r)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("n,copies,payload", [(1, 1, True), (33, 300, False), (5000, 1, True), (100_003, 3, True)])
def test_pairs(ctx, oracle, dtype, n, copies, payload):
    rng = np.random.default_rng(n)
    rk = np.repeat(np.arange(900), copies).astype(dtype)
    rng.shuffle(rk)
    rk[::400] = np.iinfo(dtype).min
    sk = rng.integers(0, 1800, n).astype(dtype)
    sk[::200] = np.iinfo(dtype).min
    ids = rng.permutation(n).astype(np.int32)
    eb, ep = (oracle.join_pairs_i64 if dtype == np.int64 else oracle.join_pairs)(rk, sk)
    t = ctx.join_build(dev(rk), dev(np.ones(len(rk), np.int32)) if payload else None)
    for rows in (None, ids):
        b, p, cnt = ctx.join_probe_pairs(t, dev(sk), len(eb) + 3, probe_rows=None if rows is None else dev(rows))
        ctx.sync()
        m = int(host(cnt)[0])
        want = ep if rows is None else rows[ep]
        assert sorted(zip(host(b)[:m].tolist(), host(p)[:m].tolist())) == sorted(zip(eb.tolist(), want.tolist()))
    if len(eb) > 1:  # a capacity one short is reported, the count is still whole
        b, p, cnt = ctx.join_probe_pairs(t, dev(sk), len(eb) - 1)
        with pytest.raises(abi.GbjError) as e:
            ctx.sync()
        assert e.value.code == abi.ERR_CAPACITY and int(host(cnt)[0]) == len(eb)
    t.destroy()
