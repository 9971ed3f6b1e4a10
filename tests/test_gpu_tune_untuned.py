"""A tuned call takes at most what the untuned one takes (with a margin for
timing): the untuned plan is among those tried."""
import numpy as np
import pytest
import torch

from gpu_util import CONFIG2_AGGS, dev, host

pytestmark = pytest.mark.gpu


def best_ms(f):
    f()
    best = float("inf")
    for _ in range(25):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


# the fewest partitions are 2, 4 and 8 times too few here: 2.1, 1.3 and 1.3 times the time
@pytest.mark.parametrize("nb,np_", [(1 << 14, 1 << 22), (1 << 16, 1 << 20), (1 << 18, 1 << 24)])
def test_radix_join(ctx, nb, np_):
    rng = np.random.default_rng(nb)
    bk, pk = dev(rng.permutation(nb).astype(np.int32)), dev(rng.integers(0, nb, np_).astype(np.int32))
    run = lambda: ctx.radix_join_agg(bk, None, pk, None, CONFIG2_AGGS)  # noqa: E731
    ctx.tune_clear()
    try:
        untuned, exp = best_ms(run), host(run()).tolist()
        ctx.autotune_radix_join(bk, None, pk, None, CONFIG2_AGGS)
        assert best_ms(run) < 1.2 * untuned
        assert host(run()).tolist() == exp
    finally:
        ctx.tune_clear()


def test_groupby(ctx):
    rng = np.random.default_rng(4)
    k, v = dev(rng.integers(0, 5000, 1 << 22).astype(np.int32)), dev(rng.integers(0, 9, 1 << 22).astype(np.int32))
    run = lambda: ctx.groupby(k, v, 5000, expected_groups=5000)  # noqa: E731
    ctx.tune_clear()
    try:
        untuned = best_ms(run)
        ctx.autotune_groupby(k, v, 5000)
        assert best_ms(run) < 1.2 * untuned
        assert int(host(run()[5])[0]) == 5000
    finally:
        ctx.tune_clear()
