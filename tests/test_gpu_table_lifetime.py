"""A table destroyed right behind a probe that still waits on its stream: the
table's memory must not go to work on another stream before that probe has
read it.  The pool has no room beside the table, so that the other stream's
request is for that memory."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host
from proteus_gb300 import abi, engine

pytestmark = pytest.mark.gpu

AGGS = {"xor": [(abi.AGG_COUNT, abi.VAL_ONE), (abi.AGG_SUM, abi.VAL_ROWID_XOR)],
        "list": [(abi.AGG_COUNT, abi.VAL_ONE), (abi.AGG_SUM, abi.VAL_BUILD), (abi.AGG_MAX, abi.VAL_PROBE)]}
N, DELAY = 1 << 19, 40_000_000  # clock cycles: some 20 ms


@pytest.fixture
def small():
    c = engine.Context(0, pool_bytes=24 << 20)
    yield c
    torch.cuda.synchronize()
    c.close()


@pytest.mark.parametrize("streams", [1, 2])
@pytest.mark.parametrize("aggs", ["xor", "list", "pairs"])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_destroy_behind_a_probe(small, oracle, dtype, aggs, streams):
    rng = np.random.default_rng(3)
    n = N
    rk = rng.permutation(n).astype(dtype)
    rp = rng.integers(-1000, 1000, n).astype(np.int32)
    sk = rng.integers(0, n + n // 8, 4 * n).astype(dtype)
    sp = rng.integers(-1000, 1000, 4 * n).astype(np.int32)
    # the other stream's work: a sort, whose scratch is cleared and written
    cols = [dev(rng.integers(0, 1 << 30, 700_000).astype(np.int32)) for _ in range(2)]
    d = [dev(c) for c in (rk, rp, sk, sp)]
    side = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for s in side:
        with torch.cuda.stream(s):  # their first launches, and the second stream's kernels loaded
            torch.cuda._sleep(1000)
            small.sort_by_key(cols, 0)
    torch.cuda.synchronize()
    with torch.cuda.stream(side[0]):
        t = small.join_build(d[0], d[1])
    side[0].synchronize()
    outs = []
    for s in side[:streams]:
        with torch.cuda.stream(s):
            torch.cuda._sleep(DELAY)
            if aggs == "pairs":
                outs.append(small.join_probe_pairs(t, d[2], 4 * n))
            else:
                outs.append(small.join_probe_agg(t, d[2], d[3], AGGS[aggs]))
    t.destroy()
    with torch.cuda.stream(side[2]):
        got = small.sort_by_key(cols, 0)
    torch.cuda.synchronize()
    small.sync()
    key, by = host(cols[0]), host(got[0])
    assert (by == np.sort(key)).all()
    if aggs == "pairs":
        for b, p, cnt in outs:
            m = int(host(cnt)[0])
            assert m == int((sk < n).sum())
            assert (rk[host(b)[:m]] == sk[host(p)[:m]]).all()
    else:
        fn = oracle.join_agg if dtype == np.int32 else oracle.join_agg_i64
        exp = fn(rk, rp, sk, sp, AGGS[aggs])
        for o in outs:
            assert host(o).tolist() == exp
