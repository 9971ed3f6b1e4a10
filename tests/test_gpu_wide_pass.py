"""One-pass partitioning on 9 to 12 bits: tile edges, ragged ends, every digit
function, column and pair output, all keys in one partition, against the
oracle's clusters and the two-pass partition."""
import numpy as np
import pytest

from gpu_util import CONFIG2_AGGS, cpu_threads, dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_payload", [True, False])  # tiles of 8192 and 12288 tuples
@pytest.mark.parametrize("digit,shift", [(abi.DIGIT_HASH, 0), (abi.DIGIT_KEY, 20), (abi.DIGIT_HASH, 19)])
@pytest.mark.parametrize("n,bits", [(1, 9), (8191, 10), (8193, 9), (12288, 12), (12289, 11), (152 * 12288 + 5, 12)])
def test_partition(ctx, oracle, n, bits, digit, shift, with_payload):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(-(1 << 31), 1 << 31, n).astype(np.int32)
    if n == 8193:
        keys[:] = 12345  # one partition takes all
    pay = rng.integers(-10**6, 10**6, n).astype(np.int32) if with_payload else None
    ok, op, off = ctx.partition(dev(keys), dev(pay) if with_payload else None, bits, shift=shift, digit=digit)
    ctx.sync()
    ek, ep, eoff = oracle.radix_cluster(keys, pay, shift, bits, digit == abi.DIGIT_HASH)
    assert (host(off).astype(np.uint64) == eoff).all()
    part = np.repeat(np.arange(1 << bits), np.diff(eoff.astype(np.int64)))
    for k, p in ((host(ok), host(op)), (ek, ep)):  # tuples keep no order inside a partition
        order = np.lexsort((p, k, part))
        k[:], p[:] = k[order], p[order]
        if k is not ek:
            got = k.copy(), p.copy()
    assert (got[0] == ek).all() and (got[1] == ep).all()


@pytest.mark.parametrize("nr,ns", [(3, 70_000), (40_000, 1 << 20), (4_000_000, 4_000_001), (17_000_000, 17_000_000)])
def test_join_plans(ctx, oracle, nr, ns):
    """The automatic bits and kernel shape of small, ordinary and large sides
    against a pinned two-pass plan."""
    rng = np.random.default_rng(nr)
    rk = rng.permutation(nr).astype(np.int32) * 5
    sk = rng.integers(0, 2 * nr, ns).astype(np.int32) * 5
    cols = dev(rk), None, dev(sk), None
    got = host(ctx.radix_join_agg(*cols, CONFIG2_AGGS)).tolist()
    assert got == host(ctx.radix_join_agg(*cols, CONFIG2_AGGS, bits=13, passes=2, block=512)).tolist()
    if ns < 1 << 21:
        assert got == oracle.radix_join_agg(rk, None, sk, None, CONFIG2_AGGS, threads=cpu_threads())
