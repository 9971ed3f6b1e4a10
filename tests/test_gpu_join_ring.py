"""The two-aggregate lists over a table that is more than a third full (probes that go on to the next bucket wait in
the warp's ring) and over sparser ones, at probe counts around a warp's tile, against the oracle."""
import numpy as np
import pytest

from gpu_util import dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu
COUNT = (abi.AGG_COUNT, abi.VAL_ONE)


@pytest.mark.parametrize("n_build", [40, 11_000, 16_000])  # load 0.63 (smallest table), 0.34, 0.49
@pytest.mark.parametrize("copies", [1, 7])
@pytest.mark.parametrize("payload", [False, True])
@pytest.mark.parametrize("n_probe,offset", [(1, 0), (31, 0), (127, 1), (128, 0), (129, 0), (4 * 128 + 5, 3), (700_001, 0),
                                            (700_001, 1)])
def test_probe_ring(ctx, oracle, n_build, copies, payload, n_probe, offset):
    rng = np.random.default_rng(n_probe + n_build)
    low = np.iinfo(np.int32).min
    rk = (rng.permutation(n_build) // copies * 3).astype(np.int32)
    rk[::n_build // 2] = low
    rp = rng.integers(low, -low, n_build).astype(np.int32)
    sk = rng.integers(-30, 3 * n_build // copies + 30, n_probe + offset).astype(np.int32)
    sk[offset::37] = low
    sp = rng.integers(low, -low, n_probe + offset).astype(np.int32)
    t = ctx.join_build(dev(rk), dev(rp) if payload else None)
    dk, dp = dev(sk)[offset:], dev(sp)[offset:]
    for op in (abi.VAL_PRODUCT, abi.VAL_ROWID_XOR)[0 if payload else 1:]:  # a product takes a payload
        aggs = [COUNT, (abi.AGG_SUM, op)]
        got = host(ctx.join_probe_agg(t, dk, dp, aggs)).tolist()
        assert got == oracle.join_agg(rk, rp if payload else None, sk[offset:], sp[offset:], aggs)
    ctx.sync()
    t.destroy()
