"""The kernel timing's names are those of the kernels that ran."""
import numpy as np
import pytest

from gpu_util import CONFIG1_AGGS, dev
from proteus_gb300 import abi

pytestmark = pytest.mark.gpu

LIST = [(abi.AGG_COUNT, abi.VAL_ONE), (abi.AGG_MIN, abi.VAL_PROBE)]


# build rows: the table (a power of two from twice the rows) a third full or less, or more
@pytest.mark.parametrize("dtype,n,call,name", [
    (np.int32, 5000, "product", "k_jb_probe_agg"), (np.int32, 8000, "product", "k_jb_probe_ring"),
    (np.int32, 8000, "list", "k_jb_probe_list"), (np.int64, 8000, "product", "k_jb_probe_list"),
    (np.int32, 8000, "pairs", "k_jb_probe_list"), (np.int64, 8000, "pairs", "k_jb_probe_list")])
def test_probe(ctx, dtype, n, call, name):
    k, p = dev(np.arange(n, dtype=dtype)), dev(np.arange(n, dtype=np.int32))
    t = ctx.join_build(k, p)
    ctx.profile(True)
    try:
        if call == "pairs":
            ctx.join_probe_pairs(t, k, n)
        else:
            ctx.join_probe_agg(t, k, p, LIST if call == "list" else CONFIG1_AGGS)
        ctx.sync()
        probes = [x for x in ctx.profile_dump() if x.startswith("k_jb_probe")]
    finally:
        ctx.profile(False)
    assert probes == [name]
    t.destroy()
