"""Build sides around the table that one CTA makes in shared memory (at most
4096 rows, or fewer with a larger table asked for): every probe form, copies of
a key, full buckets, the lowest key, an empty side, against the oracle."""
import numpy as np
import pytest

from gpu_util import CONFIG1_AGGS, CONFIG2_AGGS, dev, host
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu

LIST = [(abi.AGG_SUM, abi.VAL_BUILD_ROWID), (abi.AGG_MIN, abi.VAL_BUILD_KEY), (abi.AGG_COUNT, abi.VAL_ONE)]


@pytest.mark.parametrize("n,hash_bits", [(0, 0), (1, 0), (31, 0), (33, 6), (1025, 0), (2048, 13), (2048, 14), (4096, 0),
                                         (4097, 0)])
@pytest.mark.parametrize("keys", ["unique", "copies", "one"])
@pytest.mark.parametrize("with_payload", [True, False])
def test_small_build(ctx, oracle, n, hash_bits, keys, with_payload):
    rng = np.random.default_rng(n)
    if keys == "unique":
        rk = rng.permutation(n).astype(np.int32) * 3
    else:
        rk = rng.integers(0, max(1, n // 40), n).astype(np.int32) if keys == "copies" else np.full(n, 7, np.int32)
    rk[::17] = np.iinfo(np.int32).min
    rp = rng.integers(-1000, 1000, n).astype(np.int32) if with_payload else None
    sk = rng.integers(0, max(2, 3 * n), 3001).astype(np.int32)
    sk[::50] = np.iinfo(np.int32).min
    sk[1::50] = 7
    sp = rng.integers(-1000, 1000, len(sk)).astype(np.int32)
    t = ctx.join_build(dev(rk), dev(rp) if with_payload else None, hash_bits=hash_bits)
    for aggs in ([CONFIG1_AGGS] if with_payload else []) + [CONFIG2_AGGS, LIST]:
        got = host(ctx.join_probe_agg(t, dev(sk), dev(sp), aggs)).tolist()
        ctx.sync()
        assert got == oracle.join_agg(rk, rp, sk, sp, aggs)
    eb, ep = oracle.join_pairs(rk, sk)
    b, p, cnt = ctx.join_probe_pairs(t, dev(sk), len(eb) + 1)
    ctx.sync()
    m = int(host(cnt)[0])
    assert m == len(eb)
    assert sorted(zip(host(b)[:m].tolist(), host(p)[:m].tolist())) == sorted(zip(eb.tolist(), ep.tolist()))
    t.destroy()
