"""Build sides with copies of their keys: few keys with many rows, groups of a
warp's lanes with one key around the size from which they are placed together,
tables in shared memory and in L2, against the oracle; and what copies cost."""
import numpy as np
import pytest
import torch

from gpu_util import CONFIG1_AGGS, CONFIG2_AGGS, dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu

LIST = [(abi.AGG_SUM, abi.VAL_BUILD_ROWID), (abi.AGG_MIN, abi.VAL_BUILD_KEY), (abi.AGG_COUNT, abi.VAL_ONE)]


# run: neighbouring rows with one key, so as many lanes of a warp (7, 8, 32 among them)
@pytest.mark.parametrize("n,distinct,run", [(4096, 1, 1), (4000, 2, 1), (4096, 16, 1), (3333, 1111, 1), (8192, 4096, 2),
                                            (6000, 1, 1), (20_000, 300, 7), (20_000, 300, 8), (40_000, 900, 32),
                                            (1 << 16, 1 << 14, 1), (100_000, 50_000, 9), (1 << 18, 1 << 18, 1)])
@pytest.mark.parametrize("with_payload", [True, False])
def test_copies(ctx, oracle, n, distinct, run, with_payload):
    rng = np.random.default_rng(n + distinct)
    keys = rng.integers(-(1 << 31) + 1, 1 << 31, distinct)
    rk = np.repeat(keys[rng.permutation(-(-n // run)) % distinct], run)[:n].astype(np.int32)
    rp = rng.integers(-1000, 1000, n).astype(np.int32) if with_payload else None
    sk = np.concatenate([rng.choice(keys, 500), rng.integers(-(1 << 31), 1 << 31, 500)]).astype(np.int32)
    sp = rng.integers(-1000, 1000, len(sk)).astype(np.int32)
    for _ in range(3):
        t = ctx.join_build(dev(rk), dev(rp) if with_payload else None)
        for aggs in ([CONFIG1_AGGS] if with_payload else []) + [CONFIG2_AGGS, LIST]:
            got = host(ctx.join_probe_agg(t, dev(sk), dev(sp), aggs)).tolist()
            ctx.sync()
            assert got == oracle.join_agg(rk, rp, sk, sp, aggs)
        t.destroy()


def build_ms(ctx, k):
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        t = ctx.join_build(k, k)
        b.record()
        torch.cuda.synchronize()
        t.destroy()
        best = min(best, a.elapsed_time(b))
    return best


# against unique keys: 42 and 3.0 times now, 280 and 7.6 when every slot on the way was claimed
@pytest.mark.parametrize("n,distinct,times", [(4000, 2, 100), (4_000_000, 250_000, 5)])
def test_what_copies_cost(ctx, n, distinct, times):
    k = dev(np.random.default_rng(2).permutation(n).astype(np.int32))
    assert build_ms(ctx, k % distinct) < times * build_ms(ctx, k)
