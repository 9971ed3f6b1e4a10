"""A filter destroyed right behind a probe that still waits on its stream (see
test_gpu_table_lifetime.py): its memory goes to other streams behind that probe."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host
from proteus_gb300 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streams", [1, 2])
def test_destroy_behind_a_probe(lib, streams):
    ctx = engine.Context(0, pool_bytes=22 << 20)
    rng = np.random.default_rng(5)
    size = 1 << 27  # positions: 16 MiB
    keys = rng.integers(0, size, 100_000).astype(np.int32)
    probe = np.concatenate([rng.permutation(keys), rng.integers(0, size, 300_000).astype(np.int32)])
    exp = np.flatnonzero(np.isin(probe, keys))
    cols = [dev(rng.integers(0, 1 << 30, 700_000).astype(np.int32)) for _ in range(2)]
    dk, dp = dev(keys), dev(probe)
    side = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for s in side:
        with torch.cuda.stream(s):
            torch.cuda._sleep(1000)
            ctx.sort_by_key(cols, 0)
    torch.cuda.synchronize()
    with torch.cuda.stream(side[0]):
        f = ctx.bloom_build(dk, size)
    side[0].synchronize()
    outs = []
    for s in side[:streams]:
        with torch.cuda.stream(s):
            torch.cuda._sleep(40_000_000)  # clock cycles: some 20 ms
            outs.append(ctx.bloom_probe(f, dp))
    ctx.bloom_destroy(f)
    with torch.cuda.stream(side[2]):
        got = ctx.sort_by_key(cols, 0)
    torch.cuda.synchronize()
    ctx.sync()
    assert (host(got[0]) == np.sort(host(cols[0]))).all()
    for rows, cnt in outs:
        m = int(host(cnt)[0])
        assert (host(rows)[:m] == exp).all() and m == len(exp)
    ctx.close()
