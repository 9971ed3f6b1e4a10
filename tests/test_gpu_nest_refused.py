"""More int64 groups than a table takes: found without going round all of a
table that has four times the slots, so a refusal costs what it costs in the
least table."""
import numpy as np
import pytest
import torch

from gpu_util import dev
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu


def refused_ms(ctx, d, least):
    ctx.sync()
    if least:  # room for 8192 slots, not for 32,768
        ctx.set_pool_limit(ctx.pool_stats()["in_use"] + 48 * 8193 + 1024)
    best = float("inf")
    try:
        for _ in range(3):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            ctx.nest_i64(d, d, 16, expected_groups=3000)
            b.record()
            with pytest.raises(abi.GbjError) as e:
                ctx.sync()
            assert e.value.code == abi.ERR_CAPACITY
            best = min(best, a.elapsed_time(b))
    finally:
        ctx.set_pool_limit(0)
    return best


def test_refusal_is_no_dearer_in_a_larger_table(ctx):
    d = dev(np.random.default_rng(1).permutation(1 << 19))
    assert refused_ms(ctx, d, False) < 2 * refused_ms(ctx, d, True)


@pytest.mark.parametrize("n", [8193, 9000, 20_000])
def test_every_count_past_the_limit(ctx, n):
    """Just past the limit the walks still end in empty slots: the emit refuses."""
    d = dev(np.repeat(np.arange(n, dtype=np.int64) << 20, 60))
    ctx.nest_i64(d, d, n, expected_groups=3000)
    with pytest.raises(abi.GbjError) as e:
        ctx.sync()
    assert e.value.code == abi.ERR_CAPACITY
