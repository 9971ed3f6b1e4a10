"""A pool block asked for while calls on the context's own stream still use the
pool: what is written into it on another stream must not reach their scratch."""
import ctypes as C

import numpy as np
import pytest
import torch

from gpu_util import dev, host
from proteus_gb300 import engine

pytestmark = pytest.mark.gpu


def test_block_beside_running_sorts(lib):
    ctx = engine.Context(0, pool_bytes=20 << 20)  # a sort of 700,000 rows takes 12 MB of it
    n = 700_000
    rng = np.random.default_rng(6)
    cols = [dev(rng.integers(0, 1 << 30, n).astype(np.int32)) for _ in range(2)]
    rows = dev(np.arange(n, dtype=np.int32))
    exp = np.argsort(host(cols[0]), kind="stable")
    side = torch.cuda.Stream()
    for _ in range(10):
        outs = [[torch.empty_like(c) for c in cols] for _ in range(8)]
        torch.cuda.synchronize()
        for out in outs:  # on the context's own stream
            ins = (C.c_void_p * 2)(*[c.data_ptr() for c in cols])
            ous = (C.c_void_p * 2)(*[o.data_ptr() for o in out])
            ctx.check(lib.gbj_sort_by_key(ctx.handle, ins, 2, n, 0, 0, ous, None))
        blocks = []
        for _ in range(4):  # 11 MB: some of the scratch's place
            p = C.c_void_p()
            ctx.check(lib.gbj_pool_alloc(ctx.handle, 4 * n, C.byref(p)))
            ctx.check(lib.gbj_gather(ctx.handle, cols[1].data_ptr(), rows.data_ptr(), n, p, side.cuda_stream))
            blocks.append(p)
        torch.cuda.synchronize()
        for p in blocks:
            ctx.check(lib.gbj_pool_free(ctx.handle, p))
        for out in outs:
            for o, c in zip(out, cols):
                assert (host(o) == host(c)[exp]).all()
    ctx.close()
