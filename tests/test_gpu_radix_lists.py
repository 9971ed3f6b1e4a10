"""The partitioned join's accumulators and rings: aggregate lists of every
length and both specialised ones, row counts around a warp, copies of a build
key inside one bucket and over many, and the hash that marks an empty slot,
against the oracle."""
import numpy as np
import pytest

from gpu_util import CONFIG1_AGGS, CONFIG2_AGGS, cpu_threads, dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu

PAYLOADS = [(abi.AGG_SUM, abi.VAL_BUILD), (abi.AGG_MIN, abi.VAL_PROBE), (abi.AGG_MAX, abi.VAL_PRODUCT),
            (abi.AGG_COUNT, abi.VAL_ONE), (abi.AGG_MIN, abi.VAL_BUILD_KEY), (abi.AGG_OR, abi.VAL_PROBE),
            (abi.AGG_AND, abi.VAL_BUILD), (abi.AGG_SUM, abi.VAL_BUILD_KEY)]
BOTH = [(abi.AGG_SUM, abi.VAL_BUILD), (abi.AGG_SUM, abi.VAL_BUILD_ROWID), (abi.AGG_MAX, abi.VAL_ROWID_XOR)]
LISTS = {"product": CONFIG1_AGGS, "xor": CONFIG2_AGGS, "one": PAYLOADS[:1], "four": PAYLOADS[:4],
         "five": PAYLOADS[:5], "eight": PAYLOADS, "rows": BOTH}


def unmix(h):
    """The key whose 32-bit murmur3 finaliser is h."""
    h ^= h >> 16
    h = h * 0x7ED1B41D & 0xFFFFFFFF
    h ^= (h >> 13) ^ (h >> 26)
    h = h * 0xA5CB9243 & 0xFFFFFFFF
    h ^= h >> 16
    return np.uint32(h).astype(np.int32)


@pytest.mark.parametrize("block", [512, 1024])
@pytest.mark.parametrize("name", LISTS)
@pytest.mark.parametrize("nr,ns,copies,bits", [(1, 1, 1, 1), (33, 4097, 1, 1), (5000, 100_003, 1, 2),
                                               (20_000, 30_001, 3, 3), (9000, 9000, 900, 1)])
def test_lists(ctx, oracle, block, name, nr, ns, copies, bits):
    rng = np.random.default_rng(nr + ns)
    # the keys go up from one whose hash is the empty marker
    keys = np.arange(max(1, nr // copies), dtype=np.int32) * 7 + unmix(0x80000000)
    rk = keys[np.arange(nr) % len(keys)]
    rng.shuffle(rk)
    sk = keys[rng.integers(0, len(keys), ns)] + rng.integers(0, 2, ns).astype(np.int32)
    sk[0] = keys[0]
    rp, sp = (rng.integers(-1000, 1000, n).astype(np.int32) for n in (nr, ns))
    aggs = LISTS[name]
    got = host(ctx.radix_join_agg(dev(rk), dev(rp), dev(sk), dev(sp), aggs, bits=bits, block=block)).tolist()
    ctx.sync()
    assert got == oracle.join_agg(rk, rp, sk, sp, aggs, threads=cpu_threads())


def test_product_over_many_partitions(ctx, oracle):
    rng = np.random.default_rng(2)
    rk = rng.permutation(3_000_017).astype(np.int32)
    sk = rng.integers(0, 6_000_034, 4_000_001).astype(np.int32)
    rp, sp = rng.integers(0, 1000, len(rk)).astype(np.int32), rng.integers(0, 1000, len(sk)).astype(np.int32)
    got = host(ctx.radix_join_agg(dev(rk), dev(rp), dev(sk), dev(sp), CONFIG1_AGGS)).tolist()
    assert got == oracle.join_agg(rk, rp, sk, sp, CONFIG1_AGGS, threads=cpu_threads())
