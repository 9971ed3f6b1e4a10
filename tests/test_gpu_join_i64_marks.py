"""int64 join tables at their fullest (half of the slots taken), where rows go
past buckets while others write them: every mark, payload and row id has to
survive, so each build is repeated and every aggregate compared with the oracle."""
import numpy as np
import pytest

from gpu_util import dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu

AGGS = [(abi.AGG_COUNT, abi.VAL_ONE), (abi.AGG_SUM, abi.VAL_BUILD), (abi.AGG_SUM, abi.VAL_BUILD_ROWID),
        (abi.AGG_SUM, abi.VAL_ROWID_XOR), (abi.AGG_SUM, abi.VAL_PRODUCT), (abi.AGG_MIN, abi.VAL_BUILD),
        (abi.AGG_MAX, abi.VAL_BUILD)]


@pytest.mark.parametrize("copies", [1, 2, 3, 7])
@pytest.mark.parametrize("n", [32, 1 << 12, 1 << 17])
def test_displaced_rows(ctx, oracle, n, copies):
    rng = np.random.default_rng(n + copies)
    distinct = np.unique(rng.integers(-(1 << 62), 1 << 62, (n + copies - 1) // copies))
    rk = rng.permutation(np.resize(distinct, n))
    rp = rng.integers(-(1 << 31), 1 << 31, n).astype(np.int32)
    sk = np.concatenate([distinct, distinct ^ 1, rng.choice(distinct, n)])
    sp = rng.integers(-1000, 1000, len(sk)).astype(np.int32)
    exp = oracle.join_agg_i64(rk, rp, sk, sp, AGGS)
    d = [dev(c) for c in (rk, rp, sk, sp)]
    for _ in range(8):
        t = ctx.join_build(d[0], d[1])
        assert t.slots == 2 * n
        out = ctx.join_probe_agg(t, d[2], d[3], AGGS)
        ctx.sync()
        assert host(out).tolist() == exp
        t.destroy()
