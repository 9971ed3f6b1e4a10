"""The serving probe at the edges of its sectors, rings and items: tables with
long runs, copies of build keys within and across sectors, the lowest key on
both sides, groups in shared and in global memory, more matches of a group than
the shared sums hold, against the oracle."""
import numpy as np
import pytest

from gpu_util import dev
from proteus_gb300 import abi, serve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [3, 900, 5000])
@pytest.mark.parametrize("n_build,copies,n_probe", [(1, 1, 33), (511, 1, 4097), (512, 500, 2000), (40_000, 3, 70_001),
                                                    (2000, 1, 300_007)])
@pytest.mark.parametrize("resident", [False, True])
def test_probe(ctx, oracle, groups, n_build, copies, n_probe, resident):
    rng = np.random.default_rng(n_build + groups)
    bk = (np.arange(n_build) // copies * 7 - 1000).astype(np.int32)
    rng.shuffle(bk)
    bk[::300] = np.iinfo(np.int32).min
    bg = rng.integers(0, groups, n_build).astype(np.int32) * 1_000_003
    pk = rng.choice(np.concatenate([bk, bk + 1]), n_probe).astype(np.int32)
    pv = rng.integers(-(1 << 31), 1 << 31, n_probe).astype(np.int32)
    if n_probe == 300_007:
        pk[:200_000] = bk[1]  # one group takes more than 65535 matches
    cols = [dev(a) for a in (bk, bg, pk, pv)]
    srv = serve.Server(ctx, max_batch=4, max_inflight=2)
    out = serve.Output(groups + 1)
    if resident:
        t = srv.register_table(cols[0], cols[1], groups)
        ticket = srv.submit(None, None, cols[2], cols[3], groups, out, table=t)
    else:
        ticket = srv.submit(*cols, groups, out)
    assert srv.wait(ticket, timeout=60.0) == abi.OK
    for got, exp in zip(out.sorted(), oracle.join_groupby(bk, bg, pk, pv)[:3]):
        assert len(got) == len(exp) and (got == exp).all()
    srv.close()
